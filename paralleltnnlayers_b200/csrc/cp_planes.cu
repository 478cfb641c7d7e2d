// CP4 and three-factor CP convolutions (3x3, pad 1) and their factor gradients as products over whole rank planes.
//
//   P[r] = sum_c K1[c,r] X[c]      Z[r]  = stencil(P[r])       U[t]  = sum_r K0[t,r] Z[r]
//   Q[r] = sum_t K0[t,r] dU[t]     Zt[r] = stencil^T(Q[r])     dX[c] = sum_r K1[c,r] Zt[r]
//   dK0[t,r] = sum_px dU[t] Z[r]   dK1[c,r] = sum_px X[c] Zt[r]   dS[y,x,r] = sum_px Q[r] P[r] shifted by (y-1, x-1)
//
// The tile kernels do the three phases of a convolution one after the other in each CTA, on tiles of one image: with
// many ranks or channels, small images, or widths the row kernels do not take, a CTA is one long serial chain with idle
// lanes (64 images of 512 x 7x7 at R = 64: 51 us per convolution, 208 us for the factor gradients, for 0.1 GMAC per
// product; here 23 us and 39 us).  Here a phase is a launch of its own, over the pixels of all images as one flat range, so that a tile is
// always full and the sum can be split over a cluster; the planes (R of C channels) pass through L2.  The launches are
// programmatic dependents of one another.  The products and the factor gradients exist on FFMA and on the tensor cores, where a
// value is three bf16 parts (24 bits) and a product six of theirs; the stencils are FFMA.
// Formulas: Cuda_kernels/cp4Conv2dForward.cu:42-134, cp4Conv2dBackwardData.cu:29-109, cp4Conv2dBackwardFilter.cu:64-257.
#include <algorithm>
#include <cstdlib>
#include <type_traits>

#include "b200cp_test.h"
#include "cluster_util.cuh"
#include "common.cuh"
#include "cp_planes.cuh"
#include "mma_util.cuh"
#include "tc_common.cuh"

namespace b200cp {

std::atomic<int> g_planes_test{-1};
__device__ int g_planes_status = 0;  // 0 ok; otherwise (1 << 16) | (block index & 0xffff): a bounded wait ran out

namespace {

constexpr int kThreads = 128;

__device__ __forceinline__ float4 lds4(const float* p) { return *reinterpret_cast<const float4*>(p); }

__device__ __forceinline__ void fma4(float (&d)[4], float a, const float4& b) {
  d[0] = fmaf(a, b.x, d[0]);
  d[1] = fmaf(a, b.y, d[1]);
  d[2] = fmaf(a, b.z, d[2]);
  d[3] = fmaf(a, b.w, d[3]);
}

// ---- out[n][m][p] = sum_k F(m, k) in[n][k][p] --------------------------------------------------------------------------
// AK false: F is [K][M] (channels to ranks); true: F is [M][K] (ranks to channels).  A warp forms 4*TM rows x 32 pixels,
// TM x 4 per lane (4 row groups x 8 pixel quads): three shared-memory wavefronts per 32 FFMA at TM = 8.  128 threads per
// CTA, four and more CTAs per SM.
struct PlaneProduct {
  const float* F;
  const float* in;
  float* out;
  int M, K, mtiles, kper;
  int vecF, vecIn, vecOut;
};
struct PlaneGemm {
  PlaneProduct p[2];
  int HW, Q, maxmt, splits;     // Q = N * HW
};
constexpr int kGK = 16, kGS = 3;

template <int TM, int WM, int WN, bool AK>
__global__ void __launch_bounds__(kThreads) plane_gemm_kernel(const __grid_constant__ PlaneGemm g) {
  constexpr int BM = 4 * TM * WM, BN = 32 * WN, PA = AK ? kGK + 4 : BM;
  constexpr int kAF = AK ? BM * PA : kGK * PA, kStage = kAF + kGK * BN;
  static_assert(WM * WN == 4 && kGS * kStage >= BM * BN, "");
  __shared__ __align__(16) float smem[kGS * kStage];
  const PlaneProduct& a = g.p[blockIdx.z / g.splits];
  const int mt = blockIdx.x % g.maxmt, q0 = (blockIdx.x / g.maxmt) * BN;
  if (mt >= a.mtiles) {     // (the other product of the launch has more row tiles; a whole cluster leaves)
    grid_dependency_wait();
    return;
  }
  const int m0 = mt * BM, kb = (blockIdx.z % g.splits) * a.kper, ke = min(a.K, kb + a.kper);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, wm = warp / WN, wn = warp % WN;
  const int ty = lane >> 3, tx = lane & 7;
  const unsigned sbase = (unsigned)__cvta_generic_to_shared(smem);
  // this thread's pixel column of a stage
  constexpr int G4 = BN / 4, R4 = kThreads / G4, R1 = kThreads / BN;
  const int col = a.vecIn ? (tid % G4) * 4 : tid % BN, row0 = a.vecIn ? tid / G4 : tid / BN;
  const bool colin = q0 + col < g.Q;
  const int n = colin ? (q0 + col) / g.HW : 0, p = colin ? q0 + col - n * g.HW : 0;
  const float* in = a.in + (size_t)n * a.K * g.HW + p;

  // Every thread copies the same column of each stage, so its address runs and what is outside M or the pixels is a copy
  // of no bytes (zero fill); only the last stage of a K that is no multiple of the stage looks at k.
  const float* inp = in + (size_t)(kb + row0) * g.HW;
  auto load_in = [&](int st, int k0) {
    const unsigned d = sbase + (unsigned)(st * kStage + kAF + row0 * BN + col) * 4u;
    const float* src = inp;
    inp += (size_t)kGK * g.HW;
    const bool full = k0 + kGK <= ke;
    if (a.vecIn) {
      const size_t inc = (size_t)R4 * g.HW;
#pragma unroll
      for (int i = 0; i < kGK / R4; ++i, src += inc) {
        const bool v = colin && (full || k0 + row0 + i * R4 < ke);
        mma::cp_async16_s(d + (unsigned)(i * R4 * BN) * 4u, v ? src : a.in, v ? 16 : 0);
      }
    } else if (full && q0 + BN <= g.Q) {
      const size_t inc = (size_t)R1 * g.HW;
#pragma unroll
      for (int i = 0; i < kGK / R1; ++i, src += inc) mma::cp_async4_s(d + (unsigned)(i * R1 * BN) * 4u, src, 4);
    } else {
      const size_t inc = (size_t)R1 * g.HW;
#pragma unroll
      for (int i = 0; i < kGK / R1; ++i, src += inc) {
        const bool v = colin && k0 + row0 + i * R1 < ke;
        mma::cp_async4_s(d + (unsigned)(i * R1 * BN) * 4u, v ? src : a.in, v ? 4 : 0);
      }
    }
  };
  auto load_f = [&](int st, int k0) {
    const unsigned d0 = sbase + (unsigned)(st * kStage) * 4u;
    // groups of 4 floats or single floats along the contiguous index; ROWS threads apart along the other
    const auto copy = [&](auto width) {
      constexpr int V = decltype(width)::value, COLS = (AK ? kGK : BM) / V, ROWS = AK ? BM : kGK, RT = kThreads / COLS;
      const int c = (tid % COLS) * V, r0 = tid / COLS, ld = AK ? a.K : a.M;
      const int kc = AK ? k0 + c : m0 + c, kr = AK ? m0 + r0 : k0 + r0;
      const bool cin = kc < (AK ? ke : a.M);
      const int rend = AK ? a.M : ke;
      const float* src = a.F + (size_t)kr * ld + kc;
      const size_t inc = (size_t)RT * ld;
      unsigned d = d0 + (unsigned)(r0 * PA + c) * 4u;
#pragma unroll
      for (int i = 0; i < (ROWS + RT - 1) / RT; ++i, src += inc, d += (unsigned)(RT * PA) * 4u) {
        if (ROWS % RT && r0 + i * RT >= ROWS) break;
        const bool v = cin && kr + i * RT < rend;
        if (V == 4) mma::cp_async16_s(d, v ? src : a.F, v ? 16 : 0);
        else mma::cp_async4_s(d, v ? src : a.F, v ? 4 : 0);
      }
    };
    if (a.vecF) copy(std::integral_constant<int, 4>{});
    else copy(std::integral_constant<int, 1>{});
  };

  float acc[TM][4];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  const int steps = ke > kb ? (ke - kb + kGK - 1) / kGK : 0;
  for (int s = 0; s < kGS - 1; ++s)
    if (s < steps) load_f(s, kb + s * kGK);
  grid_dependency_wait();
  for (int s = 0; s < kGS - 1; ++s) {
    if (s < steps) load_in(s, kb + s * kGK);
    mma::cp_async_commit();
  }
  for (int s = 0; s < steps; ++s) {
    mma::cp_async_wait<kGS - 2>();
    __syncthreads();
    const int nx = s + kGS - 1;
    if (nx < steps) {
      load_f(nx % kGS, kb + nx * kGK);
      load_in(nx % kGS, kb + nx * kGK);
    }
    mma::cp_async_commit();
    const float* As = smem + (s % kGS) * kStage;
    const float* Bs = As + kAF + wn * 32 + tx * 4;
#pragma unroll
    for (int k = 0; k < kGK; k += 4) {
      if (AK) {
        float4 f[TM];
#pragma unroll
        for (int i = 0; i < TM; ++i) f[i] = lds4(As + (wm * 4 * TM + ty + 4 * i) * PA + k);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float4 b = lds4(Bs + (k + u) * BN);
#pragma unroll
          for (int i = 0; i < TM; ++i) fma4(acc[i], u == 0 ? f[i].x : u == 1 ? f[i].y : u == 2 ? f[i].z : f[i].w, b);
        }
      } else {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float4 b = lds4(Bs + (k + u) * BN);
#pragma unroll
          for (int i = 0; i < TM; i += 4) {
            const float4 f = lds4(As + (k + u) * PA + wm * 4 * TM + ty * TM + i);
            fma4(acc[i], f.x, b);
            fma4(acc[i + 1], f.y, b);
            fma4(acc[i + 2], f.z, b);
            fma4(acc[i + 3], f.w, b);
          }
        }
      }
    }
  }
  mma::cp_async_wait<0>();
  grid_launch_dependents();
  if (g.splits > 1) {
    __syncthreads();
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int m = wm * 4 * TM + (AK ? ty + 4 * i : ty * TM + i);
      *reinterpret_cast<float4*>(smem + m * BN + wn * 32 + tx * 4) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    }
    cluster_sum(smem, BM * BN, g.splits, tid, kThreads, [&](int i, float v) {
      const int m = m0 + i / BN, q = q0 + i % BN;
      if (m < a.M && q < g.Q) {
        const int nn = q / g.HW;
        a.out[((size_t)nn * a.M + m) * g.HW + (q - nn * g.HW)] = v;
      }
    });
    return;
  }
  // this thread's four pixels
  const int q = q0 + wn * 32 + tx * 4;
  size_t o[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int nn = (q + j) / g.HW;
    o[j] = (size_t)nn * a.M * g.HW + (q + j - nn * g.HW);
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + wm * 4 * TM + (AK ? ty + 4 * i : ty * TM + i);
    if (m >= a.M) continue;
    float* d = a.out + (size_t)m * g.HW;
    if (a.vecOut) {
      if (q < g.Q) *reinterpret_cast<float4*>(d + o[0]) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (q + j < g.Q) d[o[j]] = acc[i][j];
    }
  }
}

// ---- out[n][m][p] = sum_k F(m, k) in[n][k][p] on the tensor cores ---------------------------------------------------------
// The products of a CP convolution with whole rank planes: P = K1^T X (F is [K][M]) and U = K0 Z (AK: F is [M][K]).  Every value is
// three bf16 parts and a product six of theirs, as in the gradients of gemm_tc.cu: channels and ranks may differ in scale by any
// factor (that of a rank is free to move between the factor matrices).  Accumulators of 64 terms.
//
// 128 pixels are the rows of the tensor-core tile, one per TMEM lane and G threads: each loads 64 / G values of a chunk (the
// lanes of a warp read 32 neighbours of a plane, at any width or alignment) and writes them as swizzled operand rows itself, so no
// pass over memory is needed.  G = 2 where two CTAs fit an SM; else G = 4, and the loads run two chunks ahead.  Every chunk has
// its own accumulator in TMEM (chunks x rows <= 512 columns); at the end they are added up.  F is split once per CTA,
// which then walks the pixel tiles; where the pixels alone leave SMs idle the sum is split over a cluster instead.
//
// What bounds it is latency: before the first chunk 2.6 us (loads, split of F), per chunk 1.5 (0.5 of loads and splitting, 1.0 of products
// up to their commit), 1 for the read-out.  One elected lane issues the products, once the warp's next loads are on their way: the whole
// layer of 64 x 512 7x7 at R = 64 64.3 -> 61.9 us, 32 x 128 28x28 at R = 56 88.4 -> 84.5.  (A warp of its own for the issue: chunks of
// 1.2 us, but 96 registers instead of 125, and all else took as much longer.)  Both products of
// 64 x 256 14x14 at R = 32: P and Q 19.7 us on FFMA, 16.8 here, the outputs 17.5 and 15.0; of 16 x 256 -> 384 27x27 at R = 50: 39.8 and
// 34.0, 40.2 and 16.4.  Fp16 pairs with an exponent per pixel and chunk took 2 to 5 % less, and lost the result where a rank is scaled
// up in one factor and down in another (R = 24, by 2^-40 to 2^40).  Error against float64 over 60 drawn shapes 0.7 times that of FFMA.
constexpr int kTcPx = 128, kTcK = 64;
constexpr int kTcPlane = kTcPx * 128;   // bytes of one operand plane of a chunk
constexpr int kTcMaxChunks = 14;        // that fit in shared memory with rows of 32

struct PlaneTcProduct {
  const float* F;
  const float* in;
  float* out;
  int M, K, mtiles, kper;   // kper: of a CTA of the cluster, a multiple of 64
};
struct PlaneTc {
  PlaneTcProduct p[2];
  int HW, Q, maxmt, splits, pxtiles;
  int nt, chunks, cols;     // rows of a tile, a multiple of 32; chunks of a CTA; TMEM columns
  int first;                // the input is not the work of the kernel before
};

// eight values to 16 bytes of each plane
__device__ __forceinline__ void put8(uint8_t* d, uint32_t plane, const float* v) {
  tc::Bf3 w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) w[i] = tc::split3(v[2 * i], v[2 * i + 1]);
#pragma unroll
  for (int q = 0; q < 3; ++q) *reinterpret_cast<uint4*>(d + q * plane) = make_uint4(w[0].p[q], w[1].p[q], w[2].p[q], w[3].p[q]);
}
// the six products of a chunk of 16 kk terms, the smallest first
template <int KK>
__device__ __forceinline__ void mma_chunk(uint32_t d, uint64_t a, uint64_t A1, uint64_t b, uint64_t B1, uint32_t idesc) {
#pragma unroll
  for (int i = 0; i < KK; ++i) {
    tc::mma_f16_ss(d, a + 2 * A1 + i * 2, b + i * 2, idesc, i > 0);
    tc::mma_f16_ss(d, a + i * 2, b + 2 * B1 + i * 2, idesc, true);
    tc::mma_f16_ss(d, a + A1 + i * 2, b + B1 + i * 2, idesc, true);
  }
#pragma unroll
  for (int i = 0; i < KK; ++i) {
    tc::mma_f16_ss(d, a + A1 + i * 2, b + i * 2, idesc, true);
    tc::mma_f16_ss(d, a + i * 2, b + B1 + i * 2, idesc, true);
  }
#pragma unroll
  for (int i = 0; i < KK; ++i) tc::mma_f16_ss(d, a + i * 2, b + i * 2, idesc, true);
}

// An infinite value has no three parts: the second is inf - inf, and every sum that meets it comes out NaN.  Such sums are formed anew in
// fp32, which gives the infinity, or the NaN, that each is.  (Sums of finite values are NaN only where fp32 overflows too.)  Out of line:
// in line, code that is fetched and not run, 3 to 5 % of a step or layer; so the step of 64 x 256 14x14 at R = 32 takes 49.8 -> 50.2 us, layers of
// 64 x 512 7x7 at R = 64 60.2 -> 60.8 and of 16 x 256 -> 384 27x27 at R = 50 91.1 -> 88.4.
__device__ __forceinline__ float sum_fp32(const float* a, size_t ia, const float* b, size_t ib, int n) {
  float v = 0.f;
  for (int k = 0; k < n && v == v; ++k) v = fmaf(a[k * ia], b[k * ib], v);
  return v;
}
template <int N>
__device__ __forceinline__ bool any_nan(const float (&x)[N]) {   // (or infinities of both signs)
  float t[N / 2];
#pragma unroll
  for (int j = 0; j < N / 2; ++j) t[j] = x[j] + x[N / 2 + j];
#pragma unroll
  for (int n = N / 4; n; n /= 2)
#pragma unroll
    for (int j = 0; j < n; ++j) t[j] += t[n + j];
  return t[0] != t[0];
}
// rows that a group of the G x 128 threads reads out, 16 at a time
template <int G>
__device__ __forceinline__ int group_row(int grp, int nt) { return (grp * nt / G + 15) / 16 * 16; }
// what this thread read out of a tile
template <bool AK, int G>
__device__ __noinline__ void plane_sums_fp32(const PlaneTc& g, int tile, float* sums) {
  const PlaneTcProduct& a = g.p[blockIdx.z / g.splits];
  const int t = threadIdx.x & 127, grp = threadIdx.x >> 7, q = tile * kTcPx + t, m0 = blockIdx.y * g.nt;
  const int kb = (blockIdx.z % g.splits) * a.kper, n = min(a.K, kb + a.kper) - kb, image = q / g.HW, p = q - image * g.HW;
  if (q >= g.Q) return;
  for (int r = group_row<G>(grp, g.nt); r < min(group_row<G>(grp + 1, g.nt), a.M - m0); ++r) {
    float* d = g.splits > 1 ? sums + r * kTcPx + t : a.out + ((size_t)image * a.M + m0 + r) * g.HW + p;
    const float* F = AK ? a.F + (size_t)(m0 + r) * a.K + kb : a.F + (size_t)kb * a.M + m0 + r;
    if (*d != *d) *d = sum_fp32(F, AK ? 1 : a.M, a.in + ((size_t)image * a.K + kb) * g.HW + p, g.HW, n);
  }
}

template <bool AK, int G>
__global__ void __launch_bounds__(G * 128, 4 / G) plane_tc_kernel(const __grid_constant__ PlaneTc g) {
  constexpr int kThreads = G * 128;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ __align__(8) uint64_t done;
  __shared__ uint32_t tmem_slot;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), grp = tid >> 7, t = tid & 127;
  const PlaneTcProduct& a = g.p[blockIdx.z / g.splits];
  const int mt = blockIdx.y;
  if (mt >= a.mtiles) {     // (the other product of the launch has more row tiles; a whole cluster leaves)
    grid_dependency_wait();
    return;
  }
  const int nt = g.nt, m0 = mt * nt, kb = (blockIdx.z % g.splits) * a.kper, ke = min(a.K, kb + a.kper);
  const int nch = ke > kb ? (ke - kb + kTcK - 1) / kTcK : 0;
  uint8_t* Bs = sm + 3 * kTcPlane;   // [chunk][plane][nt] rows of 128 bytes
  if (tid == 0) {
    tc::mbar_init(&done, 1);
    tc::fence_barrier_init();
  }
  if (warp == 0) tc::tmem_alloc(&tmem_slot, g.cols);
  // Values of this thread's pixel, their loads in flight while chunks before them are worked on.  (cp.async into the thread's own
  // row is four lanes to a bank, 4 us a chunk; 64 values at once spill, and code that runs once costs its fetch.)
  constexpr int V = kTcK / G, AHEAD = G / 2;
  struct Pixel {
    int n, p;
    bool in;
  } at, begun;            // this thread's pixel of the chunk whose loads come next, and of the last tile whose loads have begun
  int next_tile = blockIdx.x, next_c = 0;
  auto pixel = [&](int tile) {
    const int q = tile * kTcPx + t;
    Pixel x;
    x.in = tile < g.pxtiles && q < g.Q;
    x.n = x.in ? q / g.HW : 0;
    x.p = x.in ? q - x.n * g.HW : 0;
    return x;
  };
  auto load = [&](float (&v)[V]) {
    const int k0 = next_c * kTcK + grp * V, kn = ke - kb - k0;
    const float* src = a.in + ((size_t)at.n * a.K + kb + k0) * g.HW + at.p;
#pragma unroll
    for (int k = 0; k < V; ++k) v[k] = at.in && k < kn ? src[(size_t)k * g.HW] : 0.f;
    if (next_c == 0) begun = at;
    if (++next_c >= nch) {
      next_c = 0;
      at = pixel(next_tile += gridDim.x);
    }
  };
  float v[AHEAD][V];
  at = begun = pixel(next_tile);
  if (g.first)
#pragma unroll
    for (int i = 0; i < AHEAD; ++i) load(v[i]);
  // ---- F by items of eight k (lanes along the contiguous index)
  const int k8s = nch * (kTcK / 8), along = max(AK ? k8s : nt, 1), dfast = kThreads % along, dslow = kThreads / along;
  const int items = nt * k8s;
  {
    constexpr int kBatch = 4;   // items of a thread whose loads are in flight together (one after the other 0.65 us each)
    int fast = tid % along, slow = tid / along;
    for (int i = tid; i < items; i += kBatch * kThreads) {
      float f[kBatch][8];
      int r[kBatch], k8[kBatch];
#pragma unroll
      for (int b = 0; b < kBatch; ++b) {
        r[b] = AK ? slow : fast;
        k8[b] = AK ? fast : slow;
        const int m = m0 + r[b], k = kb + k8[b] * 8;
        const bool in = i + b * kThreads < items && m < a.M;
        const size_t inc = AK ? 1 : a.M;
        const float* src = AK ? a.F + (size_t)m * a.K + k : a.F + (size_t)k * a.M + m;
#pragma unroll
        for (int j = 0; j < 8; ++j) f[b][j] = in && k + j < ke ? __ldg(src + j * inc) : 0.f;
        fast += dfast;
        slow += dslow;
        if (fast >= along) { fast -= along; ++slow; }
      }
#pragma unroll
      for (int b = 0; b < kBatch; ++b) {
        if (i + b * kThreads >= items) break;
        put8(Bs + (k8[b] >> 3) * 3 * nt * 128 + r[b] * 128 + (((k8[b] & 7) ^ (r[b] & 7)) << 4), nt * 128, f[b]);
      }
    }
  }
  tc::fence_proxy_async();
  tc::tc_fence_before_sync();
  __syncthreads();
  tc::tc_fence_after_sync();
  const uint32_t tmem = tmem_slot, lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16);
  const uint64_t d0 = tc::make_smem_desc(0, 16, 1024, tc::kSwizzle128B), a0 = d0 + (tc::smem_u32(sm) >> 4);
  const uint32_t idesc = tc::make_idesc_bf16(nt);
  float* sums = reinterpret_cast<float*>(sm);     // [nt][128], for the cluster
  bool fine = true;
  int commits = 0;
  grid_dependency_wait();
  if (!g.first)
#pragma unroll
    for (int i = 0; i < AHEAD; ++i) load(v[i]);
  auto chunk = [&](int c, float (&v)[V]) {
    if (commits) fine = tc::mbar_wait(&done, (commits - 1) & 1) && fine;   // the operand rows are free
#pragma unroll
    for (int j = 0; j < V / 8; ++j) put8(sm + t * 128 + (((grp * (V / 8) + j) ^ (t & 7)) << 4), kTcPlane, v + 8 * j);
    tc::fence_proxy_async();
    __syncthreads();
    load(v);   // (not before the fence, which may wait for them; but before the products, whose issue takes longer than a load)
    if (warp == 0 && tc::elect_one()) {
      tc::tc_fence_after_sync();
      const uint32_t d = tmem + c * nt, B1 = (uint32_t)nt * 128 >> 4;
      const uint64_t b0 = d0 + (tc::smem_u32(Bs + c * 3 * nt * 128) >> 4);
      const int left = ke - kb - c * kTcK;
      if (left > 32) mma_chunk<4>(d, a0, kTcPlane >> 4, b0, B1, idesc);
      else if (left > 16) mma_chunk<2>(d, a0, kTcPlane >> 4, b0, B1, idesc);
      else mma_chunk<1>(d, a0, kTcPlane >> 4, b0, B1, idesc);
      tc::mma_commit(&done);
    }
    ++commits;
  };
  for (int tile = blockIdx.x; tile < g.pxtiles; tile += gridDim.x) {
    const Pixel px = AHEAD == 1 || nch > 1 ? begun : pixel(tile);   // (two ahead, tiles of one chunk: the next tile's)
    for (int c = 0; c < nch; ++c) {
      if (AHEAD == 1 || !(commits & 1)) chunk(c, v[0]);
      else chunk(c, v[AHEAD - 1]);
    }
    const int rows = g.splits > 1 ? nt : px.in ? a.M - m0 : 0;   // to be written
    if (commits) fine = tc::mbar_wait(&done, (commits - 1) & 1) && fine;
    tc::tc_fence_before_sync();
    __syncthreads();
    tc::tc_fence_after_sync();
    if (tile + gridDim.x >= g.pxtiles) grid_launch_dependents();
    // ---- the accumulators of the chunks, 16 rows at a time
    const size_t inc = g.splits > 1 ? kTcPx : g.HW;
    const int first = group_row<G>(grp, nt), last = group_row<G>(grp + 1, nt);
    float* dst = (g.splits > 1 ? sums + t : a.out + ((size_t)px.n * a.M + m0) * g.HW + px.p) + first * inc;
    bool nan = false;
    for (int c0 = first; c0 < last; c0 += 16) {
      float s[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) s[j] = 0.f;
      for (int c = 0; c < nch; ++c) {
        float x[16];
        tc::tmem_ld16(lanes + c * nt + c0, x);
#pragma unroll
        for (int j = 0; j < 16; ++j) s[j] += x[j];
      }
#pragma unroll
      for (int j = 0; j < 16; ++j, dst += inc)
        if (c0 + j < rows) *dst = s[j];
      nan |= any_nan(s);
    }
    if (nan) plane_sums_fp32<AK, G>(g, tile, sums);
    tc::tc_fence_before_sync();
    __syncthreads();   // the accumulators are free
    tc::tc_fence_after_sync();
  }
  if (!fine) atomicCAS(&g_planes_status, 0, (1 << 16) | (blockIdx.x & 0xffff));
  if (warp == 0) tc::tmem_dealloc(tmem, g.cols);
  if (g.splits == 1) return;
  // The sum over the cluster, a slice of the tile per CTA, in CTA order; four pixels per load and the loads from all CTAs in
  // flight (one value at a time the 128 x 128 tile took 10 us and more; one CTA after the other 5.6k cycles for 128 x 64, now 4.7k).
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  cl.sync();
  const int quads = nt * (kTcPx / 4), share = (quads + g.splits - 1) / g.splits, e0 = (int)cl.block_rank() * share;
  const int e1 = min(quads, e0 + share);
  const float* from[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) from[k] = cl.map_shared_rank(sums, min(k, g.splits - 1));
  for (int i = e0 + tid; i < e1; i += kThreads) {
    float4 y[8];
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (k < g.splits) y[k] = lds4(from[k] + (size_t)i * 4);
    float w[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (k < g.splits) { w[0] += y[k].x; w[1] += y[k].y; w[2] += y[k].z; w[3] += y[k].w; }
    const int m = m0 + i / (kTcPx / 4), q = blockIdx.x * kTcPx + i % (kTcPx / 4) * 4;
    if (m >= a.M) break;
    int nn = q / g.HW, p = q - nn * g.HW;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (q + j < g.Q) a.out[((size_t)nn * a.M + m) * g.HW + p] = w[j];
      if (++p == g.HW) { p = 0; ++nn; }
    }
  }
  cl.sync();   // nobody reads this CTA's sums any more
}

// ---- the stencils --------------------------------------------------------------------------------------------------------
// One rank and a range of units per CTA; a unit is four pixels below one another, so that the rows of the 6 x 3 window
// are shared (4.5 loads per pixel instead of 9) and the lanes read consecutive pixels at any width.  SUMS: Z from P, Zt
// from Q and the nine correlations of Q with P (partial sums per CTA); otherwise one plane per blockIdx.z.
struct PlaneStencil {
  const float* src[2];   // P, Q
  float* dst[2];         // Z, Zt
  int flip[2];
  const float *KH, *KW, *KC;
  float* sums;           // [chunks][9][R]
  int R, H, W, HB, units, per;   // HB = row groups of four per image, units = N * HB * W
};

// Ordinary loads: this grid starts while the one that writes the planes still runs, and the read-only path (__ldg) is for
// memory that nothing writes during the kernel's life.
__device__ __forceinline__ void load_window(const float* s, int h, int w, int H, int W, float (&v)[6][3]) {
#pragma unroll
  for (int y = 0; y < 6; ++y) {
    const bool row = (unsigned)(h + y - 1) < (unsigned)H;
    const float* t = s + (y - 1) * W;
    v[y][0] = row && w > 0 ? t[-1] : 0.f;
    v[y][1] = row ? t[0] : 0.f;
    v[y][2] = row && w + 1 < W ? t[1] : 0.f;
  }
}
__device__ __forceinline__ void stencil_store(const float (&v)[6][3], const float (&w)[9], float* d, int h, int H, int W) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    float z = 0.f;
#pragma unroll
    for (int i = 0; i < 9; ++i) z = fmaf(w[i], v[k + i / 3][i % 3], z);
    if (h + k < H) d[k * W] = z;
  }
}

template <bool SUMS>
__global__ void __launch_bounds__(kThreads) plane_stencil_kernel(const __grid_constant__ PlaneStencil g) {
  const int r = blockIdx.x, tid = threadIdx.x, c = SUMS ? 0 : blockIdx.z;
  float w[9];
  const bool flip = !SUMS && g.flip[c];
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    const int t = flip ? 8 - i : i;
    w[i] = g.KC ? g.KC[t * g.R + r] : g.KH[(t / 3) * g.R + r] * g.KW[(t % 3) * g.R + r];
  }
  float s[9];
#pragma unroll
  for (int i = 0; i < 9; ++i) s[i] = 0.f;
  grid_dependency_wait();
  const int ue = min(g.units, (int)(blockIdx.y + 1) * g.per);
  for (int u = blockIdx.y * g.per + tid; u < ue; u += kThreads) {
    const int row = u / g.W, x = u - row * g.W, n = row / g.HB, h = (row - n * g.HB) * 4;
    const size_t o = ((size_t)n * g.R + r) * (g.H * g.W) + h * g.W + x;
    float v[6][3];
    load_window(g.src[c] + o, h, x, g.H, g.W, v);
    stencil_store(v, w, g.dst[c] + o, h, g.H, g.W);
    if (SUMS) {
      float q[6][3], wt[9];
      load_window(g.src[1] + o, h, x, g.H, g.W, q);
#pragma unroll
      for (int i = 0; i < 9; ++i) wt[i] = w[8 - i];
      stencil_store(q, wt, g.dst[1] + o, h, g.H, g.W);
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int i = 0; i < 9; ++i)
          if (h + k < g.H) s[i] = fmaf(q[k + 1][1], v[k + i / 3][i % 3], s[i]);
    }
  }
  grid_launch_dependents();
  if (SUMS) {
    __shared__ float red[kThreads / 32][9];
#pragma unroll
    for (int i = 0; i < 9; ++i) {
#pragma unroll
      for (int d = 16; d; d >>= 1) s[i] += __shfl_xor_sync(0xffffffffu, s[i], d);
      if ((tid & 31) == 0) red[tid >> 5][i] = s[i];
    }
    __syncthreads();
    if (tid < 9) {
      float v = red[0][tid];
#pragma unroll
      for (int k = 1; k < kThreads / 32; ++k) v += red[k][tid];
      g.sums[((size_t)blockIdx.y * 9 + tid) * g.R + r] = v;
    }
  }
}

// ---- partial factor gradients: part[split][row][r] = sum over a pixel range of D[row][q] Z[r][q] ------------------------
// On the tensor cores: 128 rows of dU or X and NT ranks per CTA, K = pixels, which both operands have contiguous.  The sum runs
// over pixels and images, of which one may be any number of binades above the others and add nothing (a masked sample: zeros in the
// other operand), so no two pixels share an exponent: a value is three bf16 parts, a product six of theirs (gemm_tc.cu).  A warp takes
// a row at a time: 64 pixels, two per lane, and 4 bytes of each plane per lane.  A chunk of 64 pixels has an accumulator of
// its own in half of TMEM (two CTAs per SM); once these are used up they are added to totals in registers.
//
// What bounds it is the splitting and latency: 64 x 256 14x14 at R = 32 17.2 us on FFMA, 14.1 here; 16 x 256 -> 384 27x27 at R = 50
// (4-byte loads) 33.1 and 26.4.  Fp16 pairs with an exponent per row and 64 pixels were no faster and lost 3e-4 of the result at 7x7 images
// beside one of 1e9 without gradient.  Three CTAs per SM with half of the TMEM columns each spill (27x27: half as long again).
struct PlaneGrad {
  const float* D[2];     // dU, X
  const float* Z[2];     // Z, Zt
  float* part;
  int rows[2], mtiles[2], row0[2];
  int vecD[2], vecZ;           // (FFMA kernel)
  int R, rtiles, HW, Q, per;   // per: pixels of a split, a multiple of 64 (FFMA: 32)
  size_t nrows;          // T + C
};
constexpr int kGradThreads = 256, kGradRows = 128;

template <int NT>
struct GradTile {
  static constexpr int chunks = 256 / NT;                            // accumulators
  static constexpr int bplane = NT * 128;
  static constexpr int stage = 3 * (kTcPlane + bplane);
  static constexpr size_t smem = 1024 + (size_t)stage;               // at least the [128][NT + 1] floats of the result
};

// an entry that met an infinite value, over pixels qb .. qe - 1 of rows that the images have `dn` and `zn` of (see sum_fp32)
__device__ __noinline__ float grad_sum_fp32(const float* D, int dn, const float* Z, int zn, int HW, int qb, int qe) {
  float v = 0.f;
  for (int q = qb; q < qe && v == v;) {
    const int n = q / HW, p = q - n * HW, len = min(HW - p, qe - q);
    v += sum_fp32(D + (size_t)n * dn * HW + p, 1, Z + (size_t)n * zn * HW + p, 1, len);
    q += len;
  }
  return v;
}

// VEC: H * W is a multiple of 4 and the rows are 16-byte aligned; a lane has four neighbours of every other row instead of two of each.
// (Half of the 4300 cycles of a chunk went into addresses and 4-byte loads: gradients in a step of 64 x 256 14x14 at R = 32 16.4 -> 13.2 us,
// layer of 32 x 128 28x28 at R = 56 84.1 -> 79.8.)
template <int NT, bool VEC>
__global__ void __launch_bounds__(kGradThreads, 2) plane_grad_tc_kernel(const __grid_constant__ PlaneGrad g) {
  using T = GradTile<NT>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ __align__(8) uint64_t done;
  __shared__ uint32_t tmem_slot;
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), grp = warp >> 2;
  const int rt = blockIdx.x % g.rtiles, mi = blockIdx.x / g.rtiles, half = mi >= g.mtiles[0] ? 1 : 0;
  const int m0 = (mi - (half ? g.mtiles[0] : 0)) * kGradRows, r0 = rt * NT, rows = half ? g.rows[1] : g.rows[0];
  const int qb = blockIdx.y * g.per, qe = min(g.Q, qb + g.per);
  const float* D = (half ? g.D[1] : g.D[0]) + (size_t)m0 * g.HW;
  const float* Z = (half ? g.Z[1] : g.Z[0]) + (size_t)r0 * g.HW;
  const int arows = min(kGradRows, rows - m0), brows = min(NT, g.R - r0);
  if (tid == 0) {
    tc::mbar_init(&done, 1);
    tc::fence_barrier_init();
  }
  if (warp == 0) tc::tmem_alloc(&tmem_slot, 256);
  tc::tc_fence_before_sync();
  __syncthreads();
  tc::tc_fence_after_sync();
  const uint32_t tmem = tmem_slot, lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16);
  const uint64_t d0 = tc::make_smem_desc(0, 16, 1024, tc::kSwizzle128B);
  const uint32_t idesc = tc::make_idesc_bf16(NT);
  const int steps = qe > qb ? (qe - qb + kTcK - 1) / kTcK : 0;
  float tot[NT / 2];
#pragma unroll
  for (int j = 0; j < NT / 2; ++j) tot[j] = 0.f;
  bool fine = true;
  // eight rows at a time, the rows of D and then those of Z; the next eight (of the next chunk after the last) are on their way
  // while eight are split
  constexpr int kGroups = (kGradRows + NT) / 8, kWarps = kGradThreads / 32;
  size_t a0 = 0, a1 = 0, b0 = 0, b1 = 0;   // this lane's two pixels (VEC: the first of its four) of the chunk that is loaded
  bool in0 = false, in1 = false;
  auto pixels = [&](int s) {
    const int q = qb + s * kTcK + (VEC ? (lane & 15) * 4 : lane * 2);
    in0 = q < qe;
    const int n0 = in0 ? q / g.HW : 0, p0 = in0 ? q - n0 * g.HW : 0;
    a0 = (size_t)n0 * rows * g.HW + p0;
    b0 = (size_t)n0 * g.R * g.HW + p0;
    if (VEC) return;
    in1 = q + 1 < qe;
    const int n1 = in1 ? (q + 1) / g.HW : 0, p1 = in1 ? q + 1 - n1 * g.HW : 0;
    a1 = (size_t)n1 * rows * g.HW + p1;
    b1 = (size_t)n1 * g.R * g.HW + p1;
  };
  float x[16];   // VEC: [4 pairs of rows][4 pixels], else [8 rows][2 pixels]
  auto load_rows = [&](int i) {
    const bool isb = i >= kGradRows / 8;
    const int first = (isb ? i - kGradRows / 8 : i) * 8 + (VEC ? lane >> 4 : 0), have = isb ? brows : arows;
    const float* src = (isb ? Z : D) + (size_t)first * g.HW;
    const float *s0 = src + (isb ? b0 : a0), *s1 = src + (isb ? b1 : a1);
    if constexpr (VEC) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float4 v = first + 2 * k < have && in0 ? *reinterpret_cast<const float4*>(s0 + (size_t)(2 * k) * g.HW) : make_float4(0.f, 0.f, 0.f, 0.f);
        x[4 * k] = v.x; x[4 * k + 1] = v.y; x[4 * k + 2] = v.z; x[4 * k + 3] = v.w;
      }
    } else {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const bool row = first + k < have;
        x[2 * k] = row && in0 ? s0[(size_t)k * g.HW] : 0.f;
        x[2 * k + 1] = row && in1 ? s1[(size_t)k * g.HW] : 0.f;
      }
    }
  };
  grid_dependency_wait();
  if (steps) {
    pixels(0);
    load_rows(warp);
  }
  for (int s = 0; s < steps; ++s) {
    const int c = s % T::chunks;
    if (s) fine = tc::mbar_wait(&done, (s - 1) & 1) && fine;   // (the other CTA of the SM works meanwhile)
#pragma unroll 1
    for (int i = warp; i < kGroups; i += kWarps) {
      const bool isb = i >= kGradRows / 8;
      const int first = (isb ? i - kGradRows / 8 : i) * 8;
      float v[16];
#pragma unroll
      for (int k = 0; k < 16; ++k) v[k] = x[k];
      if (i + kWarps < kGroups) {
        load_rows(i + kWarps);
      } else if (s + 1 < steps) {
        pixels(s + 1);
        load_rows(warp);
      }
      uint8_t* d = sm + (isb ? 3 * kTcPlane : 0) + first * 128;
      const uint32_t plane = isb ? T::bplane : kTcPlane;
      if constexpr (VEC) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const tc::Bf3 w0 = tc::split3(v[4 * k], v[4 * k + 1]), w1 = tc::split3(v[4 * k + 2], v[4 * k + 3]);
          const int row = 2 * k + (lane >> 4);
          uint8_t* o = d + row * 128 + ((((lane & 15) >> 1) ^ row) << 4) + (lane & 1) * 8;
#pragma unroll
          for (int q = 0; q < 3; ++q) *reinterpret_cast<uint2*>(o + q * plane) = make_uint2(w0.p[q], w1.p[q]);
        }
      } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const tc::Bf3 w = tc::split3(v[2 * k], v[2 * k + 1]);
          uint8_t* o = d + k * 128 + (((lane >> 2) ^ k) << 4) + (lane & 3) * 4;
#pragma unroll
          for (int q = 0; q < 3; ++q) *reinterpret_cast<uint32_t*>(o + q * plane) = w.p[q];
        }
      }
    }
    tc::fence_proxy_async();
    __syncthreads();
    if (warp == 0 && tc::elect_one()) {
      tc::tc_fence_after_sync();
      const uint32_t as = tc::smem_u32(sm);
      mma_chunk<kTcK / 16>(tmem + c * NT, d0 + (as >> 4), kTcPlane >> 4, d0 + ((as + 3 * kTcPlane) >> 4), T::bplane >> 4, idesc);
      tc::mma_commit(&done);
    }
    if (c + 1 < T::chunks && s + 1 < steps) continue;
    // the accumulators, in the order of the pixels
    fine = tc::mbar_wait(&done, s & 1) && fine;
    tc::tc_fence_after_sync();
    for (int k = 0; k <= c; ++k) {
#pragma unroll
      for (int j0 = 0; j0 < NT / 2; j0 += 16) {
        float v[16];
        tc::tmem_ld16(lanes + k * NT + grp * (NT / 2) + j0, v);
#pragma unroll
        for (int j = 0; j < 16; ++j) tot[j0 + j] += v[j];
      }
    }
    tc::tc_fence_before_sync();
    __syncthreads();   // the accumulators are free
  }
  if (!fine) atomicCAS(&g_planes_status, 0, (1 << 16) | (blockIdx.x & 0xffff));
  grid_launch_dependents();
  // through shared memory, for stores along the rows
  float* tile = reinterpret_cast<float*>(sm);   // [128][NT + 1]
#pragma unroll
  for (int j = 0; j < NT / 2; ++j) tile[((warp & 3) * 32 + lane) * (NT + 1) + grp * (NT / 2) + j] = tot[j];
  tc::tc_fence_before_sync();
  const bool nan = __syncthreads_or(any_nan(tot));
  if (warp == 0) {
    tc::tc_fence_after_sync();
    tc::tmem_dealloc(tmem, 256);
  }
  float* out = g.part + ((size_t)blockIdx.y * g.nrows + (half ? g.row0[1] : 0) + m0) * g.R + r0;
  for (int i = tid; i < arows * NT; i += kGradThreads) {
    const int m = i / NT, r = i % NT;
    if (r < brows) out[(size_t)m * g.R + r] = tile[m * (NT + 1) + r];
  }
  if (nan)
    for (int i = tid; i < arows * NT; i += kGradThreads) {
      const int m = i / NT, r = i % NT;
      if (r < brows && tile[m * (NT + 1) + r] != tile[m * (NT + 1) + r])
        out[(size_t)m * g.R + r] = grad_sum_fp32(D + (size_t)m * g.HW, rows, Z + (size_t)r * g.HW, g.R, g.HW, qb, qe);
    }
}

// ---- the same on FFMA ------------------------------------------------------------------------------------------------------
// Both operands have the pixels contiguous, so a lane reads four pixels of a row at once: 8 + TN reads of 16 bytes (one
// wavefront each: the pitch of 36 floats puts eight consecutive rows on all banks) per 32*TN FFMA.  The running sum of a
// group of eight stages (256 pixels) is added to the total separately: a plain chain over thousands of pixels would round
// more than split tensor-core sums.
constexpr int kDK = 32, kDP = kDK + 4, kDS = 3;

template <int TN, int WM, int WN>
__global__ void __launch_bounds__(kThreads) plane_grad_kernel(const __grid_constant__ PlaneGrad g) {
  constexpr int BM = 32 * WM, BN = 8 * TN * WN, kStage = (BM + BN) * kDP;
  static_assert(WM * WN == 4, "");
  extern __shared__ __align__(16) float smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, wm = warp / WN, wn = warp % WN;
  const int ty = lane >> 3, tx = lane & 7;
  const int rt = blockIdx.x % g.rtiles, mi = blockIdx.x / g.rtiles, half = mi >= g.mtiles[0] ? 1 : 0;
  const int m0 = (mi - (half ? g.mtiles[0] : 0)) * BM, r0 = rt * BN, rows = half ? g.rows[1] : g.rows[0];
  const int qb = blockIdx.y * g.per, qe = min(g.Q, qb + g.per);
  const float* D = half ? g.D[1] : g.D[0];
  const float* Z = half ? g.Z[1] : g.Z[0];
  const bool vecD = half ? g.vecD[1] : g.vecD[0], vecZ = g.vecZ;
  const unsigned sbase = (unsigned)__cvta_generic_to_shared(smem);
  // rows base .. base + NB - 1 of src [n][total][HW], 32 pixels from q0 on; a full tile needs no predicates, which with
  // the 4-byte copies (H * W not a multiple of 4) are most of the instructions around the FFMA (16 x 256 -> 384 27x27 R = 50: 58 -> 35 us)
  auto load = [&](auto nb, unsigned dst, const float* src, int base, int total, int q0, bool vec) {
    constexpr int NB = decltype(nb)::value;
    const int step = vec ? kThreads / 8 : kThreads / 32, i0 = vec ? tid >> 3 : tid >> 5;
    const int col = vec ? (tid & 7) * 4 : tid & 31, q = q0 + col, n = q / g.HW;
    const float* s = src + ((size_t)n * total + base + i0) * g.HW + (q - n * g.HW);
    const size_t inc = (size_t)step * g.HW;
    unsigned d = dst + (unsigned)(i0 * kDP + col) * 4u;
    const bool qin = q < qe;
    if (vec) {
#pragma unroll
      for (int i = 0; i < NB / (kThreads / 8); ++i, s += inc, d += (kThreads / 8) * kDP * 4u) {
        const bool v = qin && base + i0 + i * (kThreads / 8) < total;
        mma::cp_async16_s(d, v ? s : src, v ? 16 : 0);
      }
    } else if (base + NB <= total && q0 + kDK <= qe) {
#pragma unroll
      for (int i = 0; i < NB / (kThreads / 32); ++i, s += inc, d += (kThreads / 32) * kDP * 4u) mma::cp_async4_s(d, s, 4);
    } else {
#pragma unroll
      for (int i = 0; i < NB / (kThreads / 32); ++i, s += inc, d += (kThreads / 32) * kDP * 4u) {
        const bool v = qin && base + i0 + i * (kThreads / 32) < total;
        mma::cp_async4_s(d, v ? s : src, v ? 4 : 0);
      }
    }
  };
  auto load_stage = [&](int st, int q) {
    const unsigned d = sbase + (unsigned)(st * kStage) * 4u;
    load(std::integral_constant<int, BM>{}, d, D, m0, rows, q, vecD);
    load(std::integral_constant<int, BN>{}, d + BM * kDP * 4u, Z, r0, g.R, q, vecZ);
  };
  float acc[8][TN], total[8][TN];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = total[i][j] = 0.f;
  auto flush = [&] {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        total[i][j] += acc[i][j];
        acc[i][j] = 0.f;
      }
  };
  const int steps = qe > qb ? (qe - qb + kDK - 1) / kDK : 0;
  grid_dependency_wait();
  for (int s = 0; s < kDS - 1; ++s) {
    if (s < steps) load_stage(s, qb + s * kDK);
    mma::cp_async_commit();
  }
  for (int s = 0; s < steps; ++s) {
    mma::cp_async_wait<kDS - 2>();
    __syncthreads();
    const int nx = s + kDS - 1;
    if (nx < steps) load_stage(nx % kDS, qb + nx * kDK);
    mma::cp_async_commit();
    const float* As = smem + (s % kDS) * kStage + (wm * 32 + ty) * kDP;
    const float* Bs = smem + (s % kDS) * kStage + (BM + wn * 8 * TN + tx) * kDP;
#pragma unroll
    for (int k = 0; k < kDK; k += 4) {
      float4 b[TN];
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = lds4(Bs + j * 8 * kDP + k);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 a = lds4(As + i * 4 * kDP + k);
#pragma unroll
        for (int j = 0; j < TN; ++j)
          acc[i][j] = fmaf(a.w, b[j].w, fmaf(a.z, b[j].z, fmaf(a.y, b[j].y, fmaf(a.x, b[j].x, acc[i][j]))));
      }
    }
    if ((s & 7) == 7) flush();
  }
  flush();
  mma::cp_async_wait<0>();
  grid_launch_dependents();
  float* out = g.part + ((size_t)blockIdx.y * g.nrows + (half ? g.row0[1] : 0)) * g.R;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int m = m0 + wm * 32 + ty + 4 * i;
    if (m >= rows) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int r = r0 + wn * 8 * TN + tx + 8 * j;
      if (r < g.R) out[(size_t)m * g.R + r] = total[i][j];
    }
  }
}

// ---- the sums of the partials, in a fixed order ----------------------------------------------------------------------------
// EPT x 32 entries x 8 groups of partials per CTA; the last CTAs turn the correlation sums into the spatial factors' gradients.
// What bounds it is the latency of its reads (9.7 MB from L2 for 512 + 512 channels at R = 64), so a thread has four partials of
// each of its entries in flight, and a CTA of the correlations two partials of all nine taps: tap after tap with a barrier each it ran for
// 20.7k cycles where the others had left after 6.2k (64 x 256 14x14 at R = 32).  Steps: that one 66.1 -> 63.0 us, 21 x 64 7x7 at R = 81
// 27.9 -> 24.1.
struct PlaneReduce {
  const float* part;     // [splits][entries]
  const float* sums;     // [chunks][9][R]
  const float *KH, *KW;  // null: the free core, whose gradient is the sums themselves
  float* dK;
  int entries, splits, chunks, R, rblocks;
};
template <int EPT>
__global__ void __launch_bounds__(256) plane_reduce_kernel(const PlaneReduce g) {
  __shared__ float red[8][9][32];
  const int x = threadIdx.x, y = threadIdx.y;
  grid_dependency_wait();
  if ((int)blockIdx.x >= g.rblocks) {   // (the correlations take longest and come first)
    const int e0 = ((int)blockIdx.x - g.rblocks) * 32 * EPT + x;
    float v[EPT];
#pragma unroll
    for (int i = 0; i < EPT; ++i) v[i] = 0.f;
#pragma unroll 4
    for (int s = y; s < g.splits; s += 8) {
      const float* src = g.part + (size_t)s * g.entries + e0;
#pragma unroll
      for (int i = 0; i < EPT; ++i)
        if (e0 + i * 32 < g.entries) v[i] += src[i * 32];
    }
#pragma unroll
    for (int i = 0; i < EPT; ++i) red[y][i][x] = v[i];
    __syncthreads();
    if (y < EPT && e0 + y * 32 < g.entries) {
      float t = red[0][y][x];
#pragma unroll
      for (int k = 1; k < 8; ++k) t += red[k][y][x];
      g.dK[e0 + y * 32] = t;
    }
    return;
  }
  const int r = (int)blockIdx.x * 32 + x;
  const bool in = r < g.R;
  float v[9];
#pragma unroll
  for (int i = 0; i < 9; ++i) v[i] = 0.f;
  if (in)
#pragma unroll 2
    for (int s = y; s < g.chunks; s += 8) {
      const float* src = g.sums + (size_t)s * 9 * g.R + r;
#pragma unroll
      for (int i = 0; i < 9; ++i) v[i] += src[(size_t)i * g.R];
    }
#pragma unroll
  for (int i = 0; i < 9; ++i) red[y][i][x] = v[i];
  __syncthreads();
  float (&tap)[9][32] = red[0];
  for (int i = y; i < 9; i += 8) {
    float t = red[0][i][x];
#pragma unroll
    for (int k = 1; k < 8; ++k) t += red[k][i][x];
    tap[i][x] = t;
  }
  __syncthreads();
  if (!in) return;
  float* d = g.dK + g.entries + r;
  if (!g.KH) {
    for (int i = y; i < 9; i += 8) d[(size_t)i * g.R] = tap[i][x];
  } else if (y < 3) {
    float v = 0.f;
    for (int j = 0; j < 3; ++j) v = fmaf(g.KW[j * g.R + r], tap[y * 3 + j][x], v);
    d[(size_t)y * g.R] = v;
  } else if (y < 6) {
    float v = 0.f;
    for (int j = 0; j < 3; ++j) v = fmaf(g.KH[j * g.R + r], tap[j * 3 + y - 3][x], v);
    d[(size_t)y * g.R] = v;
  }
}

// ---- launches --------------------------------------------------------------------------------------------------------------
bool aligned16(const void* p) { return !(reinterpret_cast<uintptr_t>(p) & 15); }

// FFMA products
int gemm_launch(PlaneGemm g, int nprod, bool ak, bool programmatic, const DeviceInfo& di, cudaStream_t st) {
  int M = 0, K = 0;
  for (int i = 0; i < nprod; ++i) {
    M = std::max(M, g.p[i].M);
    K = std::max(K, g.p[i].K);
  }
  // the smallest row tile that holds all rows, at most 64; row and pixel tiles trade off at 128 threads
  const int bm = M <= 16 ? 16 : M <= 32 ? 32 : 64, bn = bm == 64 ? 64 : 128;
  long tiles = 0;
  g.maxmt = 0;
  for (int i = 0; i < nprod; ++i) {
    PlaneProduct& p = g.p[i];
    p.mtiles = ceil_div(p.M, bm);
    g.maxmt = std::max(g.maxmt, p.mtiles);
    tiles += (long)p.mtiles * ceil_div(g.Q, bn);
    p.vecF = !((ak ? p.K : p.M) & 3) && aligned16(p.F);
    p.vecIn = !(g.HW & 3) && aligned16(p.in);
    p.vecOut = !(g.HW & 3) && aligned16(p.out);
  }
  // two CTAs of 128 threads and more per SM are needed to hide the FFMA and shared-memory latency
  g.splits = pick_cluster(tiles, K, 2 * kGK, 3 * di.sm_count);
  for (int i = 0; i < nprod; ++i) g.p[i].kper = (int)align_up((size_t)ceil_div(g.p[i].K, g.splits), kGK);
  const dim3 grid((unsigned)((long)g.maxmt * ceil_div(g.Q, bn)), 1, nprod * g.splits);
#define PLANE_GEMM(TM, WM, WN)                                                                                          \
  do {                                                                                                                 \
    if (ak) B200CP_CUDA_OK(launch_cluster(plane_gemm_kernel<TM, WM, WN, true>, grid, dim3(kThreads), 0, st, g.splits,   \
                                          programmatic, g));                                                           \
    else B200CP_CUDA_OK(launch_cluster(plane_gemm_kernel<TM, WM, WN, false>, grid, dim3(kThreads), 0, st, g.splits,     \
                                       programmatic, g));                                                              \
  } while (0)
  if (bm == 16) PLANE_GEMM(4, 1, 4);
  else if (bm == 32) PLANE_GEMM(8, 1, 4);
  else PLANE_GEMM(8, 2, 2);
#undef PLANE_GEMM
  B200CP_LAUNCH_OK("plane_gemm_kernel");
  return B200CP_OK;
}

// Rows of a tile, the cluster split and the launch.
int tc_launch(PlaneTc g, int nprod, bool ak, bool programmatic, const DeviceInfo& di, cudaStream_t st) {
  int M = 0, K = 0;
  for (int i = 0; i < nprod; ++i) {
    M = std::max(M, g.p[i].M);
    K = std::max(K, g.p[i].K);
  }
  const int pxt = ceil_div(g.Q, kTcPx), kchunks = ceil_div(K, kTcK), widest = (int)align_up(std::min(M, 256), 32);
  const auto shared = [&](int chunks, int nt) { return 1024 + 3 * (size_t)kTcPlane + (size_t)chunks * 3 * nt * 128; };
  // outputs of up to 64 ranks: half of TMEM and of shared memory, for two CTAs per SM; ranks: all of them in one tile, which reads
  // the channels once
  const bool two = ak && kchunks == 1;
  const size_t columns = two ? 256 : 512, bytes = two ? 110 * 1024 : di.smem_optin - 256;
  const auto fits = [&] { return (size_t)g.chunks * g.nt <= columns && shared(g.chunks, g.nt) <= bytes; };
  const auto narrow = [&](int least) {
    while (!fits() && g.nt > least) g.nt = (int)align_up(g.nt / 2, 32);
  };
  const auto split = [&](int splits) {
    g.splits = splits;
    g.chunks = ceil_div(kchunks, splits);
    g.nt = widest;
  };
  split(1);
  if (ak) narrow(32);
  long tiles = 0;
  for (int i = 0; i < nprod; ++i) tiles += (long)ceil_div(g.p[i].M, g.nt) * pxt;
  // a cluster where that leaves no SM idle that has two chunks to do, and for all ranks in one tile (64 at least where the CTAs of
  // the pixels would fill the GPU by themselves)
  int splits = 1;
  while (splits < 8 && ceil_div(kchunks, splits) > (tiles * splits * 2 <= di.sm_count ? 2 : kTcMaxChunks)) splits *= 2;
  split(splits);
  while (!ak) {
    if (tiles >= di.sm_count) narrow(64);
    if (fits() || g.splits == 8 || g.chunks == 1) break;
    split(g.splits * 2);
  }
  narrow(32);
  // few pixels: narrower tiles, whose part of F is split and whose sums are stored sooner
  const auto ctas = [&] {
    long n = 0;
    for (int i = 0; i < nprod; ++i) n += (long)ceil_div(g.p[i].M, g.nt) * pxt * g.splits;
    return n;
  };
  while (g.nt > 32 && ctas() * 2 <= di.sm_count) g.nt = (int)align_up(g.nt / 2, 32);
  if (g.chunks > kTcMaxChunks || shared(g.chunks, g.nt) > (size_t)di.smem_optin - 256) return fail(B200CP_ERR_UNSUPPORTED, "cp planes: %d channels", K);
  g.maxmt = 0;
  for (int i = 0; i < nprod; ++i) {
    g.p[i].mtiles = ceil_div(g.p[i].M, g.nt);
    g.p[i].kper = g.chunks * kTcK;
    g.maxmt = std::max(g.maxmt, g.p[i].mtiles);
  }
  for (g.cols = 32; g.cols < g.chunks * g.nt;) g.cols *= 2;
  g.pxtiles = pxt;
  const size_t smem = std::max<size_t>(shared(g.chunks, g.nt), g.splits > 1 ? 1024 + sizeof(float) * g.nt * kTcPx : 0);
  // a CTA per tile, or as many as are resident at once and walk the tiles
  const int per_sm = g.cols > 256 || smem > 111 * 1024 ? 1 : 2;
  const int walkers = g.splits > 1 ? pxt : std::min(pxt, std::max(1, per_sm * di.sm_count / (g.maxmt * nprod)));
  const dim3 grid((unsigned)ceil_div(pxt, ceil_div(pxt, walkers)), g.maxmt, nprod * g.splits);
#define PLANE_TC(AK, G)                                                                                                 \
  do {                                                                                                                  \
    static std::atomic<int> set[64];                                                                                    \
    B200CP_CUDA_OK(ensure_dynamic_smem(reinterpret_cast<const void*>(plane_tc_kernel<AK, G>), set, (int)smem));         \
    B200CP_CUDA_OK(launch_cluster(plane_tc_kernel<AK, G>, grid, dim3(G * 128), smem, st, g.splits, programmatic, g));   \
  } while (0)
  if (ak && per_sm == 2) PLANE_TC(true, 2);
  else if (ak) PLANE_TC(true, 4);
  else if (per_sm == 2) PLANE_TC(false, 2);
  else PLANE_TC(false, 4);
#undef PLANE_TC
  B200CP_LAUNCH_OK("plane_tc_kernel");
  return B200CP_OK;
}

// Which kernels form the products and the gradients: lines in multiply-adds (pixels x ranks x channels) per rank class, over 1300
// random shapes (1 to 64 images of 7x7 to 64x64, 16 to 512 channels) measured both ways.  Where H W is no multiple of 4, FFMA loads
// single floats.  Tensor cores / FFMA, geometric means of convolutions between these powers of two of multiply-adds:
//               20-22 22-23 23-25 25-26 26-27 27-28 28-29 29-32
//   17-32, x 4   1.17  1.09  1.14  1.06  1.08  0.92  0.89  0.84       others  1.07  1.04  1.02  0.98  0.84  0.80  0.75  0.76
//   33-64, x 4   1.14  1.00  1.04  0.96  0.93  0.93  0.77  0.73       others  0.97  0.93  0.91  0.90  0.85  0.78  0.67  0.64
//   65-128       0.88  0.84  0.86  0.75  0.78  0.82  0.79  0.68       9-16, x 4  1.05 to 1.41, others  0.80 (from 2^29) to 1.25
// Gradients, steps with them on the tensor cores / on FFMA: 33-64 ranks 0.87 to 1.01, 65-128 0.83 to 1.02, 9-16 1.00 to 1.06.  17-32
// ranks: those with 16-byte loads 0.91 to 0.96 at any size (grads_by_quads), with 4-byte loads 0.91 from 2^29 on.
std::atomic<int> g_planes_tc_test{-1};   // b200cp_test_set_planes
struct PlanesOn {
  bool products, gradients;   // on the tensor cores
};
int planes_tc_mode() {   // B200CP_PLANES_TC: 0 FFMA, 2 tensor cores, else by the rules
  static const int env = [] {
    const char* e = getenv("B200CP_PLANES_TC");
    return e && e[0] == '0' ? 0 : e && e[0] == '2' ? 2 : 1;
  }();
  const int forced = g_planes_tc_test.load(std::memory_order_relaxed);
  return forced < 0 ? env : forced;
}
// by the shape alone: one convolution, and gradients whatever their rows
PlanesOn planes_on_tensor_cores(const b200cp_tensor_shape& s) {
  const int mode = planes_tc_mode();
  // a sum in a cluster of eight; FFMA has no such limit
  const bool sums = std::max({s.T, s.C, s.Rank}) <= 8u * kTcMaxChunks * kTcK;
  if (mode != 1) return {mode == 2 && sums, mode == 2};
  const double macs = (double)s.N * s.H * s.W * s.Rank * ((double)s.C + s.T);
  if (s.Rank <= 16) return {false, false};
  const bool single = (size_t)s.H * s.W % 4 != 0;
  if (s.Rank <= 32) return {sums && macs >= (single ? 1e8 : 268435456.0), macs >= 1e9 && single};
  // few channels: half of a K stage is padding (C + T up to 32: a step 1.01 to 1.28 times as long; 33 to 64 at 33 to 64 ranks 1.00 to
  // 1.06 with 16-byte loads, 0.94 to 0.98 without, above that 0.73 to 1.01)
  if (s.Rank > 64 && s.C + s.T <= 32) return {false, false};
  // up to 1000 pixels and 33 to 64 ranks the two are even on average, and a deep sum over few tiles loses (3 x 432 -> 64 17x17 at R = 44
  // 16.4 us on FFMA, 18.5)
  if (s.Rank <= 64 && macs < 1.3e8 && (size_t)s.N * s.H * s.W < 1000) return {false, true};
  return {sums && s.C + s.T > (s.Rank > 64 || single ? 32u : 64u), true};
}
// Gradients with 16-byte loads (plane_grad_tc_kernel<.., true>; the few buffers that are not aligned have 4-byte loads there)
bool grads_by_quads(const b200cp_tensor_shape& s) {
  return planes_tc_mode() == 1 && s.Rank > 16 && (size_t)s.H * s.W % 4 == 0 && (s.Rank <= 64 || s.C + s.T > 32);
}
// Two products of about as many channels in one launch (a step) fill the GPU earlier than one does: 17 to 32 ranks, H W a multiple
// of 4, at least 96 channels, steps between 2^26 and 2^28 multiply-adds 0.84 to 0.98 times as long (64 x 256 14x14 at R = 32
// 55.6 -> 49.8 us).  Where one has more than 1.5 times the channels of the other, up to 1.25 times.
bool even_products_on_tensor_cores(const b200cp_tensor_shape& s) {
  const double most = std::max(s.C, s.T), least = std::min(s.C, s.T);
  return planes_tc_mode() == 1 && s.Rank > 16 && s.Rank <= 32 && (size_t)s.H * s.W % 4 == 0 && least >= 96 && most <= 1.5 * least &&
         most <= 8.0 * kTcMaxChunks * kTcK && (double)s.N * s.H * s.W * s.Rank * (most + least) >= 67108864.0;
}
bool two_products_on_tensor_cores(const b200cp_tensor_shape& s) {
  return planes_on_tensor_cores(s).products || even_products_on_tensor_cores(s);
}
bool grads_on_tensor_cores(const b200cp_tensor_shape& s) { return planes_on_tensor_cores(s).gradients || grads_by_quads(s); }
// Units of a CTA of the stencil with correlations: whole turns of its threads, as many as make one to four waves of the five CTAs
// that an SM has registers for the shortest, where a CTA costs one turn more.  (Eight CTAs per SM and ranges that end
// within a turn: 32 images of 28x28 at R = 56 took three turns in each of two waves for 2.2 turns of work.  Layer of 16 x 256 -> 384
// 27x27 at R = 50 95.1 -> 92.5 us; the stencils alone gain nothing.)
int stencil_range(int units, int R, int sm_count) {
  const int turns = ceil_div(units, kThreads), resident = 5 * sm_count;
  long best = 0;
  int m = 1;
  for (int waves = 1; waves <= 4; ++waves) {
    const int k = ceil_div(turns, std::max(1, std::min(waves * resident / R, 65535)));
    const long cost = (long)ceil_div(R * ceil_div(turns, k), resident) * (k + 1);
    if (best == 0 || cost < best) { best = cost; m = k; }
  }
  return m * kThreads;
}
struct GradPlan {
  bool tc;
  int bm, bn, mt0, mt1, rtiles, splits, per;   // gradient products
  int units, chunks, cper;                     // stencil ranges
};
GradPlan grad_plan(const b200cp_tensor_shape& s, int sm_count) {
  GradPlan p{};
  const int R = (int)s.Rank, Q = (int)(s.N * s.H * s.W);
  p.tc = grads_on_tensor_cores(s);
  p.bn = !p.tc && R <= 16 ? 16 : R <= 32 ? 32 : 64;
  p.bm = p.tc || p.bn < 64 ? 128 : 64;
  p.mt0 = ceil_div((int)s.T, p.bm);
  p.mt1 = ceil_div((int)s.C, p.bm);
  p.rtiles = ceil_div(R, p.bn);
  const int tiles = (p.mt0 + p.mt1) * p.rtiles;
  // two CTAs per SM, at least a chunk each; on FFMA three (shared memory) of at least two stages
  const int want = p.tc ? std::max(1, std::min({2 * sm_count / tiles, ceil_div(Q, kTcK), 65535}))
                        : std::max(1, std::min({3 * sm_count / tiles, ceil_div(Q, 2 * kDK), 65535}));
  p.per = (int)align_up((size_t)ceil_div(Q, want), p.tc ? kTcK : kDK);
  p.splits = ceil_div(Q, p.per);
  p.units = (int)s.N * ceil_div((int)s.H, 4) * (int)s.W;
  p.cper = stencil_range(p.units, R, sm_count);
  p.chunks = ceil_div(p.units, p.cper);
  return p;
}

struct Carve {
  char* base;
  size_t used = 0;
  float* take(size_t floats) {
    float* p = reinterpret_cast<float*>(base + used);
    used += align_up(floats * sizeof(float), 256);
    return p;
  }
};
struct Buffers {
  float *P = nullptr, *Q = nullptr, *Z = nullptr, *Zt = nullptr, *sums = nullptr, *part = nullptr;
};
Buffers carve(Carve& c, const b200cp_tensor_shape& s, bool P, bool Q, bool Z, bool Zt, bool grads, int sm_count) {
  const size_t plane = (size_t)s.N * s.Rank * s.H * s.W;
  Buffers b;
  if (P) b.P = c.take(plane);
  if (Q) b.Q = c.take(plane);
  if (Z) b.Z = c.take(plane);
  if (Zt) b.Zt = c.take(plane);
  if (grads) {
    const GradPlan p = grad_plan(s, sm_count);
    b.sums = c.take((size_t)p.chunks * 9 * s.Rank);
    b.part = c.take((size_t)p.splits * (s.T + s.C) * s.Rank);
  }
  return b;
}

}  // namespace

// (32-bit pixel, entry and grid indices)
bool planes_supported(const b200cp_tensor_shape& s) {
  const size_t HW = (size_t)s.H * s.W, most = std::max({s.T, s.C, s.Rank});
  return s.Y == 3 && s.X == 3 && s.pad == 1 && (size_t)s.N * (s.H + 3) * s.W < (1u << 30) && s.Rank < 65536 &&
         ((size_t)s.T + s.C) * s.Rank < (1u << 30) && (most / 16 + 1) * (s.N * HW / 64 + 1) < (1u << 30);
}

// `parts`: what the call computes (the workspace of more parts is enough for fewer)
size_t planes_workspace(const b200cp_tensor_shape& s, int parts) {
  DeviceInfo di;
  if (!planes_supported(s) || device_info(&di)) return 0;
  const bool g = parts & kPlanesGrads, fwd = (parts & kPlanesFwd) || g, bwd = (parts & kPlanesBwd) || g;
  Carve c{nullptr};
  carve(c, s, fwd && !(parts & kPlanesNoP), bwd && !(parts & kPlanesNoQ), fwd, bwd, g, di.sm_count);
  return c.used;
}

int planes_launch(const PlanesJob& j, void* ws, size_t ws_bytes, cudaStream_t st) {
  const b200cp_tensor_shape& s = *j.s;
  DeviceInfo di;
  if (int rc = device_info(&di)) return rc;
  const bool grads = j.dK != nullptr, fwd = j.U != nullptr, bwd = j.dX != nullptr;
  const bool needP = fwd || grads, needQ = bwd || grads;
  Carve c{static_cast<char*>(ws)};
  const Buffers b = carve(c, s, needP && !j.P && !j.Psave, needQ && !j.Q && !j.Qsave, needP, needQ, grads, di.sm_count);
  if (!ws || ws_bytes < c.used || !aligned16(ws))
    return fail(B200CP_ERR_WORKSPACE, "cp planes: a 16-byte aligned workspace of %zu bytes needed, %zu given", c.used, ws_bytes);
  const float* P = j.P ? j.P : j.Psave ? j.Psave : b.P;
  const float* Q = j.Q ? j.Q : j.Qsave ? j.Qsave : b.Q;
  const int R = (int)s.Rank, T = (int)s.T, C = (int)s.C, HW = (int)(s.H * s.W), NQ = (int)s.N * HW;
  bool chained = false;
  PlaneTc g{};
  g.HW = HW;
  g.Q = NQ;
  int np = 0;
  auto products = [&](bool ak, bool programmatic) {
    if (np == 2 ? two_products_on_tensor_cores(s) : planes_on_tensor_cores(s).products) {
      g.first = !programmatic;
      return tc_launch(g, np, ak, programmatic, di, st);
    }
    PlaneGemm f{};
    f.HW = HW;
    f.Q = NQ;
    for (int i = 0; i < np; ++i) {
      f.p[i].F = g.p[i].F; f.p[i].in = g.p[i].in; f.p[i].out = g.p[i].out; f.p[i].M = g.p[i].M; f.p[i].K = g.p[i].K;
    }
    return gemm_launch(f, np, ak, programmatic, di, st);
  };
  auto product = [&](const float* F, const float* in, float* out, int M, int K) {
    PlaneTcProduct& p = g.p[np++];
    p.F = F; p.in = in; p.out = out; p.M = M; p.K = K;
  };
  if (needP && !j.P) product(j.K1, j.X, j.Psave ? j.Psave : b.P, R, C);
  if (needQ && !j.Q) product(j.K0, j.dU, j.Qsave ? j.Qsave : b.Q, R, T);
  if (np) {
    if (int rc = products(false, false)) return rc;
    chained = true;
  }
  const GradPlan gp = grad_plan(s, di.sm_count);
  PlaneStencil t{};
  t.KH = j.KH; t.KW = j.KW; t.KC = j.KC;
  t.R = R; t.H = (int)s.H; t.W = (int)s.W; t.HB = ceil_div(t.H, 4); t.units = gp.units; t.per = gp.cper;
  if (grads) {
    t.src[0] = P; t.src[1] = Q; t.dst[0] = b.Z; t.dst[1] = b.Zt; t.sums = b.sums;
    B200CP_CUDA_OK(launch_kernel(plane_stencil_kernel<true>, dim3(R, gp.chunks), dim3(kThreads), 0, st, chained, t));
  } else {
    int k = 0;
    if (fwd) { t.src[k] = P; t.dst[k] = b.Z; t.flip[k++] = 0; }
    if (bwd) { t.src[k] = Q; t.dst[k] = b.Zt; t.flip[k++] = 1; }
    t.per = ceil_div(t.units, std::max(1, std::min({ceil_div(8 * di.sm_count, R), ceil_div(t.units, kThreads), 65535})));
    B200CP_CUDA_OK(launch_kernel(plane_stencil_kernel<false>, dim3(R, ceil_div(t.units, t.per), k), dim3(kThreads), 0, st, chained, t));
  }
  B200CP_LAUNCH_OK("plane_stencil_kernel");
  np = 0;
  if (fwd) product(j.K0, b.Z, j.U, T, R);
  if (bwd) product(j.K1, b.Zt, j.dX, C, R);
  if (np)
    if (int rc = products(true, true)) return rc;
  if (!grads) return B200CP_OK;
  PlaneGrad d{};
  d.D[0] = j.dU; d.D[1] = j.X; d.Z[0] = b.Z; d.Z[1] = b.Zt;
  d.part = b.part;
  d.rows[0] = T; d.rows[1] = C; d.row0[1] = T;
  d.mtiles[0] = gp.mt0; d.mtiles[1] = gp.mt1;
  d.vecZ = !(HW & 3);
  for (int i = 0; i < 2; ++i) d.vecD[i] = !(HW & 3) && aligned16(d.D[i]);
  d.R = R; d.rtiles = gp.rtiles; d.HW = HW; d.Q = NQ; d.per = gp.per;
  d.nrows = (size_t)T + C;
  const dim3 grid((gp.mt0 + gp.mt1) * gp.rtiles, gp.splits);
#define PLANE_GRAD(KERNEL, THREADS, SMEM)                                                                               \
  do {                                                                                                                 \
    static std::atomic<int> set[64];                                                                                   \
    B200CP_CUDA_OK(ensure_dynamic_smem(reinterpret_cast<const void*>(KERNEL), set, (int)(SMEM)));                      \
    B200CP_CUDA_OK(launch_kernel(KERNEL, grid, dim3(THREADS), SMEM, st, true, d));                                     \
  } while (0)
  const size_t smem = sizeof(float) * kDS * (gp.bm + gp.bn) * kDP;   // FFMA
  const bool vec = d.vecZ && d.vecD[0] && d.vecD[1] && aligned16(d.Z[0]) && aligned16(d.Z[1]);
  if (gp.tc) {
    if (gp.bn == 32 && vec) PLANE_GRAD((plane_grad_tc_kernel<32, true>), kGradThreads, GradTile<32>::smem);
    else if (gp.bn == 32) PLANE_GRAD((plane_grad_tc_kernel<32, false>), kGradThreads, GradTile<32>::smem);
    else if (vec) PLANE_GRAD((plane_grad_tc_kernel<64, true>), kGradThreads, GradTile<64>::smem);
    else PLANE_GRAD((plane_grad_tc_kernel<64, false>), kGradThreads, GradTile<64>::smem);
  } else if (gp.bn == 16) PLANE_GRAD((plane_grad_kernel<2, 4, 1>), kThreads, smem);
  else if (gp.bn == 32) PLANE_GRAD((plane_grad_kernel<4, 4, 1>), kThreads, smem);
  else PLANE_GRAD((plane_grad_kernel<4, 2, 2>), kThreads, smem);
#undef PLANE_GRAD
  B200CP_LAUNCH_OK("plane_grad_kernel");
  PlaneReduce r{};
  r.part = b.part; r.sums = b.sums; r.KH = j.KC ? nullptr : j.KH; r.KW = j.KW; r.dK = j.dK;
  r.entries = (T + C) * R; r.splits = gp.splits; r.chunks = gp.chunks; r.R = R;
  r.rblocks = ceil_div(R, 32);
  // four entries per thread where that leaves every SM two CTAs
  if (r.entries >= 128 * 2 * di.sm_count)
    B200CP_CUDA_OK(launch_kernel(plane_reduce_kernel<4>, dim3(r.rblocks + ceil_div(r.entries, 128)), dim3(32, 8), 0, st, true, r));
  else
    B200CP_CUDA_OK(launch_kernel(plane_reduce_kernel<1>, dim3(r.rblocks + ceil_div(r.entries, 32)), dim3(32, 8), 0, st, true, r));
  B200CP_LAUNCH_OK("plane_reduce_kernel");
  return B200CP_OK;
}

// Reads (and clears) the status word of the tensor-core products; the caller has synchronised the device.
int planes_device_status(int* out) {
  int v = 0, zero = 0;
  B200CP_CUDA_OK(cudaMemcpyFromSymbol(&v, g_planes_status, sizeof(int)));
  if (v) B200CP_CUDA_OK(cudaMemcpyToSymbol(g_planes_status, &zero, sizeof(int)));
  *out = v;
  return B200CP_OK;
}

int planes_forms(const b200cp_tensor_shape& s) {
  return (planes_on_tensor_cores(s).products ? 1 : 0) | (two_products_on_tensor_cores(s) ? 2 : 0) | (grads_on_tensor_cores(s) ? 4 : 0);
}

}  // namespace b200cp

extern "C" void b200cp_test_set_planes(int planes, int tensor_cores) {
  b200cp::g_planes_test.store(planes, std::memory_order_relaxed);
  b200cp::g_planes_tc_test.store(tensor_cores, std::memory_order_relaxed);
}

extern "C" int b200cp_test_planes_on_tensor_cores(const b200cp_tensor_shape* s) {
  const b200cp::PlanesOn on = b200cp::planes_on_tensor_cores(*s);
  return (on.products ? 1 : 0) | (on.gradients ? 2 : 0);
}
