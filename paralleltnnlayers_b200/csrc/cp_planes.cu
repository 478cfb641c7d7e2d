// CP4 and three-factor CP convolutions (3x3, pad 1) and their factor gradients as products over whole rank planes.
//
//   P[r] = sum_c K1[c,r] X[c]      Z[r]  = stencil(P[r])       U[t]  = sum_r K0[t,r] Z[r]
//   Q[r] = sum_t K0[t,r] dU[t]     Zt[r] = stencil^T(Q[r])     dX[c] = sum_r K1[c,r] Zt[r]
//   dK0[t,r] = sum_px dU[t] Z[r]   dK1[c,r] = sum_px X[c] Zt[r]   dS[y,x,r] = sum_px Q[r] P[r] shifted by (y-1, x-1)
//
// The tile kernels do the three phases of a convolution one after the other in each CTA, on tiles of one image: with
// many ranks or channels, small images, or widths the row kernels do not take, a CTA is one long serial chain with idle
// lanes (64 images of 512 x 7x7 at R = 64: 52 us per convolution, 77 us for the factor gradients, for 0.1 GMAC per
// product; here 31 us and 37 us).  Here a phase is a launch of its own, over the pixels of all images as one flat range, so that a tile is
// always full and the sum can be split over a cluster; the planes (R of C channels) pass through L2.  The launches are
// programmatic dependents of one another.  Everything is exact fp32 (FFMA).
// Formulas: Cuda_kernels/cp4Conv2dForward.cu:42-134, cp4Conv2dBackwardData.cu:29-109, cp4Conv2dBackwardFilter.cu:64-257.
#include <algorithm>
#include <type_traits>

#include "cluster_util.cuh"
#include "common.cuh"
#include "cp_planes.cuh"
#include "mma_util.cuh"

namespace b200cp {
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
// Both operands have the pixels contiguous, so a lane reads four pixels of a row at once: 8 + TN reads of 16 bytes (one
// wavefront each: the pitch of 36 floats puts eight consecutive rows on all banks) per 32*TN FFMA.  The running sum of a
// group of eight stages (256 pixels) is added to the total separately: a plain chain over thousands of pixels would round
// more than the split tensor-core sums this kernel replaces.
struct PlaneGrad {
  const float* D[2];     // dU, X
  const float* Z[2];     // Z, Zt
  float* part;
  int rows[2], mtiles[2], row0[2];
  int vecD[2], vecZ;
  int R, rtiles, HW, Q, per;
  size_t nrows;          // T + C
};
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
// 32 entries x 8 groups of partials per CTA; the last CTAs turn the correlation sums into the spatial factors' gradients.
struct PlaneReduce {
  const float* part;     // [splits][entries]
  const float* sums;     // [chunks][9][R]
  const float *KH, *KW;  // null: the free core, whose gradient is the sums themselves
  float* dK;
  int entries, splits, chunks, R, eblocks;
};
__global__ void __launch_bounds__(256) plane_reduce_kernel(const PlaneReduce g) {
  __shared__ float red[8][32];
  __shared__ float tap[9][32];
  const int x = threadIdx.x, y = threadIdx.y;
  grid_dependency_wait();
  auto sum = [&](const float* src, size_t stride, int n, bool in) {
    float v = 0.f;
    if (in)
#pragma unroll 4
      for (int s = y; s < n; s += 8) v += src[(size_t)s * stride];
    __syncthreads();
    red[y][x] = v;
    __syncthreads();
    if (y == 0)
#pragma unroll
      for (int k = 1; k < 8; ++k) v += red[k][x];
    return v;
  };
  if ((int)blockIdx.x < g.eblocks) {
    const int e = blockIdx.x * 32 + x;
    const float v = sum(g.part + e, g.entries, g.splits, e < g.entries);
    if (y == 0 && e < g.entries) g.dK[e] = v;
    return;
  }
  const int r = ((int)blockIdx.x - g.eblocks) * 32 + x;
  const bool in = r < g.R;
  for (int i = 0; i < 9; ++i) {
    const float v = sum(g.sums + (size_t)i * g.R + r, (size_t)9 * g.R, g.chunks, in);
    if (y == 0) tap[i][x] = v;
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

struct GradPlan {
  int bm, bn, mt0, mt1, rtiles, splits, per;   // gradient products
  int units, chunks, cper;                     // stencil ranges
};
GradPlan grad_plan(const b200cp_tensor_shape& s, int sm_count) {
  GradPlan p{};
  const int R = (int)s.Rank, Q = (int)(s.N * s.H * s.W);
  p.bn = R <= 16 ? 16 : R <= 32 ? 32 : 64;
  p.bm = p.bn == 64 ? 64 : 128;
  p.mt0 = ceil_div((int)s.T, p.bm);
  p.mt1 = ceil_div((int)s.C, p.bm);
  p.rtiles = ceil_div(R, p.bn);
  const int tiles = (p.mt0 + p.mt1) * p.rtiles;
  // three CTAs per SM (shared memory), at least two stages each
  const int want = std::max(1, std::min({3 * sm_count / tiles, ceil_div(Q, 2 * kDK), 65535}));
  p.per = (int)align_up((size_t)ceil_div(Q, want), kDK);
  p.splits = ceil_div(Q, p.per);
  p.units = (int)s.N * ceil_div((int)s.H, 4) * (int)s.W;
  const int cw = std::max(1, std::min({ceil_div(8 * sm_count, R), ceil_div(p.units, kThreads), 65535}));
  p.cper = ceil_div(p.units, cw);
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
  PlaneGemm g{};
  g.HW = HW;
  g.Q = NQ;
  int np = 0;
  auto product = [&](const float* F, const float* in, float* out, int M, int K) {
    PlaneProduct& p = g.p[np++];
    p.F = F; p.in = in; p.out = out; p.M = M; p.K = K;
  };
  if (needP && !j.P) product(j.K1, j.X, j.Psave ? j.Psave : b.P, R, C);
  if (needQ && !j.Q) product(j.K0, j.dU, j.Qsave ? j.Qsave : b.Q, R, T);
  if (np) {
    if (int rc = gemm_launch(g, np, false, false, di, st)) return rc;
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
    B200CP_CUDA_OK(launch_kernel(plane_stencil_kernel<false>, dim3(R, gp.chunks, k), dim3(kThreads), 0, st, chained, t));
  }
  B200CP_LAUNCH_OK("plane_stencil_kernel");
  np = 0;
  if (fwd) product(j.K0, b.Z, j.U, T, R);
  if (bwd) product(j.K1, b.Zt, j.dX, C, R);
  if (np)
    if (int rc = gemm_launch(g, np, true, true, di, st)) return rc;
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
  const size_t smem = sizeof(float) * kDS * (gp.bm + gp.bn) * kDP;
#define PLANE_GRAD(TN, WM, WN)                                                                                           \
  do {                                                                                                                  \
    static std::atomic<int> set[64];                                                                                    \
    B200CP_CUDA_OK(ensure_dynamic_smem(reinterpret_cast<const void*>(plane_grad_kernel<TN, WM, WN>), set, (int)smem));  \
    B200CP_CUDA_OK(launch_kernel(plane_grad_kernel<TN, WM, WN>, grid, dim3(kThreads), smem, st, true, d));              \
  } while (0)
  if (gp.bn == 16) PLANE_GRAD(2, 4, 1);
  else if (gp.bn == 32) PLANE_GRAD(4, 4, 1);
  else PLANE_GRAD(4, 2, 2);
#undef PLANE_GRAD
  B200CP_LAUNCH_OK("plane_grad_kernel");
  PlaneReduce r{};
  r.part = b.part; r.sums = b.sums; r.KH = j.KC ? nullptr : j.KH; r.KW = j.KW; r.dK = j.dK;
  r.entries = (T + C) * R; r.splits = gp.splits; r.chunks = gp.chunks; r.R = R;
  r.eblocks = ceil_div(r.entries, 32);
  B200CP_CUDA_OK(launch_kernel(plane_reduce_kernel, dim3(r.eblocks + ceil_div(R, 32)), dim3(32, 8), 0, st, true, r));
  B200CP_LAUNCH_OK("plane_reduce_kernel");
  return B200CP_OK;
}

}  // namespace b200cp
