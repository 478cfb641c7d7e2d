// Reshaped-CP conv and CP dense layer by their multiplied-out weight, where that is faster than the factored kernels.
//
// The factored form does R times the mode products one rank after the other; on the chain kernel that is a serial loop
// of R x (modes + 1) block-wide steps, one CTA per SM, and with few CTAs it is latency, not arithmetic, that it spends its
// time on (430 us for a batch of 64 through 16x16x16 -> 4x4x4 at R = 137, 16 CTAs on 148 SMs; 223 us for eight 32x32 images
// of 16 channels at R = 11).  Multiplying the weight out first costs R multiply-adds per weight entry, spread over the whole
// GPU, and leaves one plain product, whatever R is; at low ranks and large batches the factored form does several times
// less and is faster (product.cu has the rule).
//   kron_weight_kernel : W[s][f] = sum_r prod_k F_k[s_k, f_k, r]   (conv: W[c][tap][t], with S as one more mode)
//   small_gemm_kernel  : Y[m][n] = sum_k X[m][k] W[k][n]
//   small_conv_kernel  : V[n,t,h,w] = sum_{c,y,x} W[c][y,x][t] X[n,c,h+y-1,w+x-1]
// All exact fp32 (FFMA); large weights for the tensor-core product come from kron_planes_kernel.  The product kernels are programmatic dependents of the weight kernel: their CTAs are resident
// and past their set-up when the weight is done.  Formulas: Kernels/rcp_fused_nchw.cu:4-77, Kernels/dense_cp.cu:4-46.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>

#include "cluster_util.cuh"
#include "common.cuh"
#include "mma_util.cuh"
#include "tc_common.cuh"

namespace b200cp {
namespace {

// The products add up to thousands of terms per result.  One accumulator over all of them rounds like sqrt(terms): relative
// to float64 8e-7 for 4096 inputs, where the factored form, whose longest chain is ranks x one mode, has 2e-7 (R = 8).  So
// an accumulator holds about kChain terms and is then added to a total: 1.8e-7 for the same sums.  The totals are in shared
// memory, [4][threads] float4, and cost 5 % (4096 samples of 4096 -> 4096: 3.68 to 3.88 ms; 16 more registers instead would
// leave one CTA of 512 threads per SM instead of two: 4.73 ms).  A chain of at most kChain terms has none.
constexpr int kChain = 64;
template <int NT>
__device__ __forceinline__ void flush_sums(float (&acc)[4][4], float* total, int tid, bool first) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float4* t = reinterpret_cast<float4*>(total) + i * NT + tid;
    float4 v = first ? make_float4(0.f, 0.f, 0.f, 0.f) : *t;
    v.x += acc[i][0]; v.y += acc[i][1]; v.z += acc[i][2]; v.w += acc[i][3];
    *t = v;
    acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
  }
}
template <int NT>
__device__ __forceinline__ void add_totals(float (&acc)[4][4], const float* total, int tid) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float4 v = reinterpret_cast<const float4*>(total)[i * NT + tid];
    acc[i][0] += v.x; acc[i][1] += v.y; acc[i][2] += v.z; acc[i][3] += v.w;
  }
}

// ---- the weight ----------------------------------------------------------------------------------------------------------
// The modes are cut into two halves, A (first modes, slow) and B (last modes): with the half products
// A[a][r] = prod_{k in A} F_k and B[b][r] the weight is the matrix product A B^T over r.  A CTA forms a TA x 64 tile of
// it; the half products of a chunk of 32 ranks are formed in shared memory on the way (each factor entry is read by
// 64 lanes of a CTA at most, from L1).  b runs over the fast sizes of B's modes first, so that a row of the tile is
// stored in runs of their product.
// What bounds it is the shared-memory pipe, which delivers 128 bytes a clock: 4 columns x 2 rows per thread and rank took 70 cycles per rank
// and CTA (4096 x 64 at R = 137: 13.9k cycles in all).  So a thread has 8 columns and two or four rows, and groups of threads share out the
// ranks of a chunk; their sums meet at the end.  4096 -> 64 dense at R = 137 and batch 64 15.6 -> 13.6 us, 360 -> 360 at R = 249 71 -> 64.
// (8 x 8 for tiles of 64 rows spills: 720 -> 720 at R = 89 18.5 -> 21.2 us; 4 x 8 18.4.)
constexpr int kKT = 256, kTB = 64, kRC = 32;
constexpr int kron_rows(int ta) { return ta < 32 ? 2 : 4; }                        // of a thread, which has 8 columns
constexpr int kron_groups(int ta) { return kKT * kron_rows(ta) * 8 / (ta * kTB); }   // of threads, which share out the ranks of a chunk

struct KronMode {
  const float* F;
  int ns, nf;       // slow-side and fast-side sizes
  int fs, ff;       // entry (s, f) at F[(s*fs + f*ff)*R + r]
  int os, of;       // output offset per s and per f
};
struct KronGeom {
  int nA, nB;              // modes of the halves
  KronMode A[3], B[2];     // (tap +) at most two modes in A, two in B
  int SA, FA, SB, FB;      // products of the sizes
  int R, rper;             // ranks; ranks per CTA of a cluster
  int flip;                // A[0] is the tap mode, stored back to front
  int early;               // all CTAs are resident at once: the product's may be placed now
};

// entry offset (in ranks) and output offset of half-index (s, f)
__device__ __forceinline__ void half_decode(const KronMode* m, int n, int s, int f, int flip, int* entry, int* out) {
  int o = 0;
  for (int k = n - 1; k >= 0; --k) {
    const int sk = s % m[k].ns, fk = f % m[k].nf;
    s /= m[k].ns;
    f /= m[k].nf;
    entry[k] = sk * m[k].fs + fk * m[k].ff;
    o += ((flip && k == 0) ? m[k].ns - 1 - sk : sk) * m[k].os + fk * m[k].of;
  }
  *out = o;
}

constexpr int kron_tiles(int ta) {   // floats of a chunk of ranks, then of the groups' sums
  return kRC * (ta + 4 + kTB + 4) > kron_groups(ta) * ta * kTB ? kRC * (ta + 4 + kTB + 4) : kron_groups(ta) * ta * kTB;
}
template <int TA>
constexpr size_t kron_smem() {
  return sizeof(float) * (kron_tiles(TA) + ClusterSum::floats(TA * kTB));
}

template <int TA, bool TAP>
__global__ void __launch_bounds__(kKT, 2) kron_weight_kernel(const __grid_constant__ KronGeom g, float* __restrict__ W) {
  constexpr int TI = kron_rows(TA), KG = kron_groups(TA), kGT = kKT / KG;
  extern __shared__ __align__(16) float tiles[];   // kron_smem<TA>()
  float (*As)[TA + 4] = reinterpret_cast<float (*)[TA + 4]>(tiles);
  float (*Bs)[kTB + 4] = reinterpret_cast<float (*)[kTB + 4]>(tiles + kRC * (TA + 4));
  __shared__ int ea[TA][3], eb[kTB][2], oa[TA], ob[kTB];
  if (g.early) grid_launch_dependents();
  const ClusterSum shared(tiles + kron_tiles(TA), TA * kTB, gridDim.z);
  const int tid = threadIdx.x, grp = tid / kGT, gx = tid & 7, gy = tid % kGT >> 3;
  const int a0 = blockIdx.y * TA, b0 = blockIdx.x * kTB, PA = g.SA * g.FA, PB = g.SB * g.FB;
  const int rb0 = blockIdx.z * g.rper, re = min(g.R, rb0 + g.rper);
  if (tid < TA) {
    const int a = a0 + tid;
    int e[3] = {0, 0, 0}, o = 0;
    if (a < PA) half_decode(g.A, g.nA, a / g.FA, a % g.FA, g.flip, e, &o);
    ea[tid][0] = e[0]; ea[tid][1] = e[1]; ea[tid][2] = e[2];
    oa[tid] = o;
  } else if (tid >= 128 && tid < 128 + kTB) {
    const int i = tid - 128, b = b0 + i;
    int e[2] = {0, 0}, o = 0;
    if (b < PB) half_decode(g.B, g.nB, b / g.FB, b % g.FB, 0, e, &o);
    eb[i][0] = e[0]; eb[i][1] = e[1];
    ob[i] = o;
  }
  float acc[TI][8];
#pragma unroll
  for (int i = 0; i < TI; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
  // A warp fills 8 ranks x 4 rows per turn: full sectors from global memory, all banks of the transposed tile.  The
  // entries of the next chunk are fetched, all loads of a thread together, while the current one is multiplied; a mode
  // that a half does not have reads nothing and counts as 1.
  constexpr int NROW = (TA + kTB + 31) / 32, NE = NROW * (kRC / 8), NM = TAP ? 3 : 2;
  const int rl = tid & 7, row0 = (tid >> 5) * 4 + ((tid >> 3) & 3);
  __syncthreads();   // the entry offsets
  const float* src[NROW][NM];
  bool in[NROW];
#pragma unroll
  for (int i = 0; i < NROW; ++i) {
    const int row = i * 32 + row0;
    const bool inA = row < TA;
    in[i] = inA ? a0 + row < PA : row < TA + kTB && b0 + row - TA < PB;
#pragma unroll
    for (int k = 0; k < NM; ++k)
      src[i][k] = !in[i] || k >= (inA ? g.nA : g.nB) ? nullptr
                  : inA ? g.A[k].F + (size_t)ea[row][k] * g.R + rl : g.B[k % 2].F + (size_t)eb[row - TA][k % 2] * g.R + rl;
  }
  float next[NM][NE];
  auto fetch = [&](int r0) {
#pragma unroll
    for (int i = 0; i < NROW; ++i)
#pragma unroll
      for (int k = 0; k < NM; ++k)
#pragma unroll
        for (int rb = 0; rb < kRC / 8; ++rb)
          next[k][i * (kRC / 8) + rb] = !in[i] || r0 + rb * 8 + rl >= re ? 0.f : src[i][k] ? __ldg(src[i][k] + r0 + rb * 8) : 1.f;
  };
  if (rb0 < re) fetch(rb0);
  for (int r0 = rb0; r0 < re; r0 += kRC) {
    if (r0 > rb0) __syncthreads();
#pragma unroll
    for (int i = 0; i < NROW; ++i) {
      const int row = i * 32 + row0;
#pragma unroll
      for (int rb = 0; rb < kRC / 8; ++rb) {
        const int e = i * (kRC / 8) + rb;
        const float v = next[0][e] * next[1][e] * (TAP ? next[NM - 1][e] : 1.f);
        if (row < TA) As[rb * 8 + rl][row] = v;
        else if (row < TA + kTB) Bs[rb * 8 + rl][row - TA] = v;
      }
    }
    __syncthreads();
    if (r0 + kRC < re) fetch(r0 + kRC);
    const int rn = min(kRC, re - r0);
#pragma unroll 2
    for (int r = grp; r < rn; r += KG) {
      const float4 b0 = *reinterpret_cast<const float4*>(&Bs[r][gx * 4]), b1 = *reinterpret_cast<const float4*>(&Bs[r][32 + gx * 4]);
      const float b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
      float a[TI];
#pragma unroll
      for (int i = 0; i < TI; ++i) a[i] = As[r][gy * TI + i];
#pragma unroll
      for (int i = 0; i < TI; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
  }
  // Of more CTAs than SMs not earlier: CTAs of the product that start while this grid still fills up are stacked on few SMs (138 CTAs
  // of small_conv_kernel took 170 us instead of 60).
  if (!g.early) grid_launch_dependents();
  // the groups' sums, [group][TA][64]
  __syncthreads();
#pragma unroll
  for (int i = 0; i < TI; ++i) {
    float* t = tiles + (grp * TA + gy * TI + i) * kTB + gx * 4;
    *reinterpret_cast<float4*>(t) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    *reinterpret_cast<float4*>(t + 32) = make_float4(acc[i][4], acc[i][5], acc[i][6], acc[i][7]);
  }
  __syncthreads();
  const int tx = tid & 15, ty = tid >> 4;
  const auto total = [&](int row) {
    const float* t = tiles + row * kTB + tx * 4;
    float4 v = *reinterpret_cast<const float4*>(t);
#pragma unroll
    for (int q = 1; q < KG; ++q) {
      const float4 w = *reinterpret_cast<const float4*>(t + q * TA * kTB);
      v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
    }
    return v;
  };
  if (gridDim.z > 1) {   // a small weight: the CTAs of a cluster took a share of the ranks each
    shared.ready();
#pragma unroll
    for (int i = 0; i < TA / 16; ++i) {
      const float4 v = total(i * 16 + ty);
      const int o = (i * 16 + ty) * kTB + tx * 4;
      shared.put(o, v.x);
      shared.put(o + 1, v.y);
      shared.put(o + 2, v.z);
      shared.put(o + 3, v.w);
    }
    shared.sum(TA * kTB, tid, kKT, [&](int i, float v) {
      const int a = i / kTB, b = i % kTB;
      if (a0 + a < PA && b0 + b < PB) W[oa[a] + ob[b]] = v;
    });
    return;
  }
  const int b = b0 + tx * 4;
  const bool run4 = b + 3 < PB && ob[tx * 4 + 3] - ob[tx * 4] == 3 && !(ob[tx * 4] & 3);
#pragma unroll
  for (int i = 0; i < TA / 16; ++i) {
    const int row = i * 16 + ty;
    if (a0 + row >= PA) continue;
    const float4 v = total(row);
    const int o0 = oa[row];
    float* d = W + o0;
    if (run4 && !(o0 & 3)) {
      *reinterpret_cast<float4*>(d + ob[tx * 4]) = v;
    } else {
      const float w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (b + j < PB) d[ob[tx * 4 + j]] = w[j];
    }
  }
}

// ---- the weight as the operand planes of the tensor-core product (gemm_tc.cu) ------------------------------------------
// Row s of the weight gets the exponent of a bound, sum_r prod_k max_f |F_k[s_k, f, r]|, which needs no pass over the weight (it is
// some 2^5 above the largest entry; of the 18 binades below a row's largest value that keep 22 bits this costs five).
// What bounds this is latency: the largest values of all slices of the modes go to shared memory once, the loads of a thread together,
// and a row, one warp, multiplies one of each mode.  4096 x 4096 at R = 32: 5.2 us; a warp that read the slices of its row
// from global memory, eight rows per CTA, 13.5.
constexpr int kRowsEx = 32;       // rows, and warps, of a CTA
__host__ __device__ __forceinline__ const KronMode& kron_mode_of(const KronGeom& g, int k) { return k < g.nA ? g.A[k] : g.B[k - g.nA]; }

__device__ __forceinline__ float largest_of_slice(const KronMode& m, int slice, int R, int r) {
  const float* src = m.F + (size_t)slice * m.fs * R + r;
  unsigned mx = 0;
  for (int f0 = 0; f0 < m.nf; f0 += 8) {
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = __ldg(src + (size_t)(min(f0 + j, m.nf - 1) * m.ff) * R);
#pragma unroll
    for (int j = 0; j < 8; ++j) mx = max(mx, tc::abs_bits(v[j]));
  }
  return __uint_as_float(mx);
}

__global__ void __launch_bounds__(32 * kRowsEx) kron_exponent_kernel(const __grid_constant__ KronGeom g, int rows, int* __restrict__ ex) {
  extern __shared__ float largest[];   // [slice of all modes][rank]: at most 4 x 16 slices of 256 ranks
  const int lane = threadIdx.x & 31, row = blockIdx.x * kRowsEx + (threadIdx.x >> 5), order = g.nA + g.nB;
  grid_launch_dependents();
  int at[4] = {0, 0, 0, 0}, slices = 0;   // the row's slice of each mode
  for (int k = 0; k < order; ++k) slices += kron_mode_of(g, k).ns;
  for (int i = threadIdx.x; i < slices * g.R; i += 32 * kRowsEx) {
    int slice = i / g.R, k = 0;
    const int r = i - slice * g.R;
    for (; slice >= kron_mode_of(g, k).ns; ++k) slice -= kron_mode_of(g, k).ns;
    largest[i] = largest_of_slice(kron_mode_of(g, k), slice, g.R, r);
  }
  int s = row;
#pragma unroll
  for (int k = 3; k >= 0; --k)
    if (k < order) {
      const int ns = kron_mode_of(g, k).ns;
      slices -= ns;
      at[k] = slices + s % ns;
      s /= ns;
    }
  __syncthreads();
  if (row >= rows) return;
  float sum = 0.f;
  for (int r = lane; r < g.R; r += 32) {
    float prod = 1.f;
#pragma unroll
    for (int k = 3; k >= 0; --k)
      if (k < order) prod *= largest[at[k] * g.R + r];
    sum += prod;
  }
#pragma unroll
  for (int d = 16; d; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
  if (lane == 0) ex[row] = tc::row_exponent(tc::abs_bits(sum * 1.001f), tc::kLeast);
}

// 128 x 128 entries per CTA and tile on the tensor cores: the half products of 64 ranks at a time as three bf16 parts, the first of six bits
// (split3_short in tc_common.cuh), K-major, and eight products of parts, the smallest first; an accumulator of the largest has 64 ranks, that of
// the others all.  A CTA keeps A's parts, where R is at most 64, and walks the tiles of B.  A thread splits the 64 entries that it has of one row of the tile into hi and lo; through shared memory, a warp
// for itself, they are stored as runs of 64 bytes of a row.
//
// What bounds it are the phases of a tile one after the other, of which the stores take the longest (a CTA forms, multiplies and stores in 2300,
// 1300 and 5500 of 9600 cycles; two per SM overlap).  4096 x 4096, times in us at R = 4 / 32 / 64 / 100 / 256: 33 / 37 / 51 / 107 / 193, with 128 x 128
// tiles of FFMA 33 / 53 / 84 / - / 345.  Error of a layer's output against float64, of 44 layers of 4 to 256 ranks, over that with FFMA: 0.55 (256
// ranks) to 1.00 (4).  With first parts of eight bits and six products, 2 to 10 % faster, it was up to 1.08; with one accumulator for
// all products 3.3 (R = 100).
// A part is a bf16 number, whose subnormals begin at 2^-126 like those of fp32, and the third is 2^-16 of the value: so the half products are lifted by
// 2^17 and keep their 24 bits down to the smallest normal number.  Where one of a tile is above 2^43, what overflows for that (half products above
// 2^111, weights above 2^94) is formed anew in fp32 (form_entries).  Without the look at the largest and the lift: 0.5 us less at R = 32.
__device__ int g_kron_status = 0;   // 0 ok; otherwise (1 << 16) | (block index & 0xffff): a bounded wait ran out
constexpr int kPT = 128, kKeep = 256, kPart = kPT * 128;   // bytes of a part of a half: 64 ranks
constexpr float kDrop = 1.f / (tc::kLift * tc::kLift), kLarge = 5.76460752303423488e17f;   // 2^59: no sum of 256 products of less overflows
constexpr size_t kPlanesSmem = 1024 + 6 * kPart;

struct KronTile {   // entries of a half in a tile
  int e[kPT][2], o[kPT], row[kPT];   // entry of each mode (in ranks), offset and row in the weight (both add up)
};

// the entries of row a of a tile in the runs of 16 columns from c0 on that `which` has bits of; none where a half product of the row is infinite or NaN
__device__ __noinline__ void form_entries(const KronGeom& g, const KronTile& ta, const KronTile& tb, int a, int c0, int count, unsigned which, int pitch,
                                          const int* ex, __half* hi, size_t plane) {
  const float *a0 = g.A[0].F + ta.e[a][0], *a1 = g.A[g.nA - 1].F + ta.e[a][g.nA - 1];
  const auto of_row = [&](int r) { return g.nA > 1 ? a0[r] * a1[r] : a0[r]; };
  float none = 0.f;
#pragma unroll 8
  for (int r = 0; r < g.R; ++r) none = fmaf(of_row(r), 0.f, none);
  if (none != 0.f) return;
  for (int c = 0; c < count; ++c) {
    if (!(which >> (c >> 4) & 1)) continue;
    const float *b0 = g.B[0].F + tb.e[c0 + c][0], *b1 = g.B[g.nB - 1].F + tb.e[c0 + c][g.nB - 1];
    float v = 0.f;
    for (int r = 0; r < g.R && v == v; ++r) v = fmaf(of_row(r), g.nB > 1 ? b0[r] * b1[r] : b0[r], v);
    const int o = ta.o[a] + tb.o[c0 + c];
    v *= tc::exp2_int(-ex[o / pitch]);
    const __half h = __float2half_rn(v);
    hi[o] = h;
    hi[plane + o] = __float2half_rn(v - __half2float(h));
  }
}

template <bool MANY>   // more than 64 ranks
__global__ void __launch_bounds__(256, 2) kron_planes_kernel(const __grid_constant__ KronGeom g, int pitch, int btiles,
                                                          const int* ex, __half* __restrict__ hi, size_t plane, bool vec) {
  extern __shared__ __align__(16) uint8_t raw[];
  uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~uintptr_t(1023));
  __shared__ KronTile ta, tb[2];
  __shared__ __align__(8) uint64_t done;
  __shared__ uint32_t tmem_slot;
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), quarter = warp & 3, grp = warp >> 2;
  const int a0 = blockIdx.y * kPT, PA = g.SA * g.FA, PB = g.SB * g.FB;
  auto table = [&](bool isA, int first, int i, KronTile& t) {
    int e[3] = {0, 0, 0}, o = 0;
    if (isA && first + i < PA) half_decode(g.A, g.nA, (first + i) / g.FA, (first + i) % g.FA, 0, e, &o);
    if (!isA && first + i < PB) half_decode(g.B, g.nB, (first + i) / g.FB, (first + i) % g.FB, 0, e, &o);
    t.e[i][0] = e[0] * g.R; t.e[i][1] = e[1] * g.R;
    t.o[i] = o;
    t.row[i] = o / pitch;
  };
  if (tid == 0) {
    tc::mbar_init(&done, 1);
    tc::fence_barrier_init();
  }
  if (warp == 0) tc::tmem_alloc(&tmem_slot, 256);
  if (tid < kPT) table(true, a0, tid, ta);
  else table(false, blockIdx.x * kPT, tid - kPT, tb[0]);
  tc::tc_fence_before_sync();
  __syncthreads();
  tc::tc_fence_after_sync();
  const uint32_t tmem = tmem_slot, lanes = tmem + ((uint32_t)(quarter * 32) << 16);
  // the half products of ranks r0 .. r0 + 63 as parts, [row][rank]; two ranks of a row per lane, rows four apart in the halves of a warp
  // (16 bytes of a row and of the one four on are in different banks)
  auto form = [&](const KronMode* m, int n, const KronTile& t, int r0, uint8_t* dst) {   // returns the largest, NaN apart
    float most = 0.f;
    const float *f0 = m[0].F, *f1 = m[n - 1].F;
    for (int h = 0; h < 2 && r0 + h * 32 < g.R; ++h) {
      const int k = h * 32 + (lane & 15) * 2, r = r0 + k, c0 = min(r, g.R - 1), c1 = min(r + 1, g.R - 1);
#pragma unroll
      for (int i0 = 0; i0 < 8; i0 += 4) {
        float x[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int row = warp * 16 + i0 * 2 + i + (lane >> 4) * 4;
          const float *p = f0 + t.e[row][0], *q = f1 + t.e[row][n - 1];
          x[i][0] = p[c0]; x[i][1] = p[c1]; x[i][2] = q[c0]; x[i][3] = q[c1];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int row = warp * 16 + i0 * 2 + i + (lane >> 4) * 4;
          const float p = x[i][0] * tc::kLift, q = x[i][1] * tc::kLift, u = n > 1 ? p * x[i][2] : p, v = n > 1 ? q * x[i][3] : q;
          most = tc::most_of(most, u, v);
          const tc::Bf3 w = tc::split3_short<true>(r < g.R ? u : 0.f, r + 1 < g.R ? v : 0.f);
          uint8_t* d = dst + row * 128 + ((((k >> 3) ^ row) & 7) << 4) + (k & 7) * 2;
#pragma unroll
          for (int j = 0; j < 3; ++j) *reinterpret_cast<uint32_t*>(d + j * kPart) = w.p[j];
        }
      }
    }
    return most;
  };
  const uint64_t d0 = tc::make_smem_desc(0, 16, 1024, tc::kSwizzle128B);
  constexpr uint32_t idesc = tc::make_idesc_bf16(kPT);
  const int srow = ta.row[quarter * 32 + lane];
  bool fine = true;
  int waits = 0;
  float most_a = 0.f;
  if (!MANY) most_a = form(g.A, g.nA, ta, 0, sm);
  int turn = 0;
  for (int bt = blockIdx.x; bt < btiles; bt += gridDim.x, turn ^= 1) {
    const int b0 = bt * kPT;
    const KronTile& t = tb[turn];
    float tot[MANY ? 64 : 1];
    bool large = false;
    int scale[4];   // exponents of this lane's row in the first column of each 16
    for (int r0 = 0; r0 < (MANY ? g.R : 1); r0 += 64) {
      if (MANY) most_a = form(g.A, g.nA, ta, r0, sm);
      const float most = fmaxf(most_a, form(g.B, g.nB, t, r0, sm + 3 * kPart));
      tc::fence_proxy_async();
      large = __syncthreads_or(most >= kLarge) || (r0 && large);
      if (warp == 0 && tc::elect_one()) {
        tc::tc_fence_after_sync();
        const uint64_t ad = d0 + (tc::smem_u32(sm) >> 4), bd = ad + (3 * kPart >> 4), p1 = kPart >> 4;
        const int steps = min(4, (g.R - r0 + 15) / 16);
        for (int k = 0; k < steps; ++k) {
          tc::mma_f16_ss(tmem + kPT, ad + 2 * p1 + k * 2, bd + p1 + k * 2, idesc, r0 > 0 || k > 0);
          tc::mma_f16_ss(tmem + kPT, ad + p1 + k * 2, bd + 2 * p1 + k * 2, idesc, true);
          tc::mma_f16_ss(tmem + kPT, ad + 2 * p1 + k * 2, bd + k * 2, idesc, true);
          tc::mma_f16_ss(tmem + kPT, ad + k * 2, bd + 2 * p1 + k * 2, idesc, true);
          tc::mma_f16_ss(tmem + kPT, ad + p1 + k * 2, bd + p1 + k * 2, idesc, true);
          tc::mma_f16_ss(tmem + kPT, ad + p1 + k * 2, bd + k * 2, idesc, true);
          tc::mma_f16_ss(tmem + kPT, ad + k * 2, bd + p1 + k * 2, idesc, true);
          tc::mma_f16_ss(tmem, ad + k * 2, bd + k * 2, idesc, k > 0);
        }
        tc::mma_commit(&done);
      }
      __syncwarp();
      if (r0 == 0 && tid >= kPT) table(false, (bt + gridDim.x) * kPT, tid - kPT, tb[turn ^ 1]);
      if (!MANY || r0 + 64 >= g.R) {
        grid_dependency_wait();
#pragma unroll
        for (int q = 0; q < 4; ++q) scale[q] = ex[srow + t.row[grp * 64 + q * 16]];
      }
      fine = tc::mbar_wait(&done, waits++ & 1) && fine;   // (the other CTA of the SM works meanwhile)
      __syncwarp();
      tc::tc_fence_after_sync();
      if constexpr (MANY) {
#pragma unroll
        for (int j0 = 0; j0 < 64; j0 += 16) {
          float v[16];
          tc::tmem_ld16(lanes + grp * 64 + j0, v);
#pragma unroll
          for (int j = 0; j < 16; ++j) tot[j0 + j] = r0 ? tot[j0 + j] + v[j] : v[j];
        }
        tc::tc_fence_before_sync();
      }
    }
    uint8_t* stage = sm + 3 * kPart + warp * 4096;   // [hi | lo][32 rows][64 bytes], B is used up
    unsigned bad = 0;   // runs of 16 columns with an entry that is not finite
#pragma unroll
    for (int j0 = 0; j0 < 64; j0 += 32) {
      const int c0 = grp * 64 + j0;
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int cq = c0 + q * 16;
        float v[16], w[16];
        if constexpr (MANY) {
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = tot[j0 + q * 16 + j];
        } else {
          tc::tmem_ld16(lanes + cq, v);
        }
        tc::tmem_ld16(lanes + kPT + cq, w);
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] += w[j];
        if (large) {
          float most = 0.f;
#pragma unroll
          for (int j = 0; j < 16; j += 2) most = tc::most_nan(most, v[j], v[j + 1]);
          if (!(most <= FLT_MAX)) bad |= 1u << (j0 / 16 + q);
        }
        if (t.row[cq] == t.row[cq + 15]) {   // one row of the weight (b's rows do not descend; columns past the end have row 0)
          const float sc = kDrop * tc::exp2_int(-scale[j0 / 16 + q]);   // (2^-148 at least)
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] *= sc;
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] *= kDrop * tc::exp2_int(-ex[srow + t.row[cq + j]]);
        }
        uint32_t h[8], l[8];
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
          const __half2 a = __floats2half2_rn(v[j], v[j + 1]);
          const float2 f = __half22float2(a);
          const __half2 b = __floats2half2_rn(v[j] - f.x, v[j + 1] - f.y);
          h[j / 2] = *reinterpret_cast<const uint32_t*>(&a);
          l[j / 2] = *reinterpret_cast<const uint32_t*>(&b);
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint8_t* d = stage + lane * 64 + (((q * 2 + c) ^ (lane >> 1)) & 3) * 16;
          *reinterpret_cast<uint4*>(d) = make_uint4(h[c * 4], h[c * 4 + 1], h[c * 4 + 2], h[c * 4 + 3]);
          *reinterpret_cast<uint4*>(d + 2048) = make_uint4(l[c * 4], l[c * 4 + 1], l[c * 4 + 2], l[c * 4 + 3]);
        }
      }
      __syncwarp();
      const int c = c0 + (lane & 3) * 8, left = PB - (b0 + c), ob = t.o[c];
      const bool run8 = vec && left >= 8 && t.o[c + 7] - ob == 7, run4 = left >= 4 && t.o[c + 3] - ob == 3, next4 = left >= 8 && t.o[c + 7] - t.o[c + 4] == 3;
      uint4 hs[4], ls[4];
      int oas[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int row = i * 8 + (lane >> 2);
        const uint8_t* src = stage + row * 64 + (((lane & 3) ^ (row >> 1)) & 3) * 16;
        hs[i] = *reinterpret_cast<const uint4*>(src);
        ls[i] = *reinterpret_cast<const uint4*>(src + 2048);
        oas[i] = ta.o[quarter * 32 + row];
      }
      // Rows of odd length begin anywhere: where the lanes' runs are not on a grid of four, a lane has a column and the warp a row at a time (a lane's
      // eight values one by one are a sector each: 14x11x11 -> 12x15x12 at R = 21 54 us, this way 25, FFMA 39).
      bool grid4 = run4 && next4;
#pragma unroll
      for (int i = 0; i < 4; ++i) grid4 = grid4 && !((oas[i] + ob) & 3) && !((oas[i] + t.o[c + 4]) & 3);
      if (!__all_sync(0xffffffffu, left <= 0 || grid4)) {
        const int col = c0 + lane, oc = t.o[col];
#pragma unroll 4
        for (int row = 0; row < 32; ++row) {
          const uint8_t* src = stage + row * 64 + (((lane >> 3) ^ (row >> 1)) & 3) * 16 + (lane & 7) * 2;
          const int o = ta.o[quarter * 32 + row] + oc;
          if (a0 + quarter * 32 + row < PA && b0 + col < PB) {
            hi[o] = *reinterpret_cast<const __half*>(src);
            hi[plane + o] = *reinterpret_cast<const __half*>(src + 2048);
          }
        }
        __syncwarp();
        continue;
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int a = quarter * 32 + i * 8 + (lane >> 2), oa = oas[i], o = oa + ob;
        const uint4 h = hs[i], l = ls[i];
        if (a0 + a >= PA) continue;
        if (run8 && !(o & 7)) {
          *reinterpret_cast<uint4*>(hi + o) = h;
          *reinterpret_cast<uint4*>(hi + plane + o) = l;
          continue;
        }
        if (left <= 0) continue;
        const int o4 = oa + t.o[c + 4];
        *reinterpret_cast<uint2*>(hi + o) = make_uint2(h.x, h.y);
        *reinterpret_cast<uint2*>(hi + plane + o) = make_uint2(l.x, l.y);
        *reinterpret_cast<uint2*>(hi + o4) = make_uint2(h.z, h.w);
        *reinterpret_cast<uint2*>(hi + plane + o4) = make_uint2(l.z, l.w);
      }
      __syncwarp();   // (an entry formed anew replaces what another lane has stored)
    }
    if (bad && a0 + quarter * 32 + lane < PA)
      form_entries(g, ta, t, quarter * 32 + lane, grp * 64, min(64, PB - b0 - grp * 64), bad, pitch, ex, hi, plane);
    tc::tc_fence_before_sync();
    __syncthreads();   // the accumulators and B are free, the table of the next tile written
  }
  if (!fine) atomicCAS(&g_kron_status, 0, (1 << 16) | (blockIdx.x & 0xffff));
  if (warp == 0) {
    tc::tc_fence_after_sync();
    tc::tmem_dealloc(tmem, 256);
  }
}

// ---- Y[M][N] = X[M][K] W[K][N] -------------------------------------------------------------------------------------------
// CTA tile BM x BN, 4 x 4 results per thread; KG groups of threads share the K rows of a stage (a small tile has few
// results, so the threads are spread over K instead).  The CTAs of a cluster split K further.
constexpr int kGStages = 3;
template <int BM, int BN>
struct GemmTile {
  static constexpr int NT = BM == 64 || BM == 16 ? 512 : 256;     // 16 warps hide the FFMA and shared-memory latency that 8 do not
  static constexpr int KG = NT * 16 / (BM * BN);      // 64x64 -> 2, 32x64 -> 2, 16x64 -> 8, 16x32 -> 16, 8x32 -> 16
  static constexpr int BK = KG > 2 ? 64 : 32;         // K rows of a stage
  static constexpr int PA = BK + 4;
  static constexpr int stage = BM * PA + BK * (BN + 4);
  static constexpr int flush = kChain / (BK / KG);    // stages of an accumulator
  static constexpr int buf = kGStages * stage > KG * BM * BN ? kGStages * stage : KG * BM * BN;
  static bool is_long(int kper) { return (kper + BK - 1) / BK > flush; }
  static size_t smem(int kper) { return sizeof(float) * ((size_t)buf + (is_long(kper) ? 16 * NT : 0) + ClusterSum::floats(BM * BN)); }
};

// LONG: more than kChain terms per accumulator (4096 -> 64 at batch 64, whose chains are short enough, 12.6 us without the totals and 12.9 with)
template <int BM, int BN, bool VECA, bool LONG>
__global__ void __launch_bounds__(GemmTile<BM, BN>::NT) small_gemm_kernel(const float* __restrict__ X, const float* __restrict__ W,
                                                         float* __restrict__ Y, int M, int N, int K, int ldw, int kper,
                                                         int splits) {
  using T = GemmTile<BM, BN>;
  constexpr int kBN = BN, kGT = T::NT, TXN = BN / 4;
  extern __shared__ __align__(16) float smem[];
  const int tid = threadIdx.x;
  const int kg = tid / (kGT / T::KG), gt = tid - kg * (kGT / T::KG), tx = gt % TXN, ty = gt / TXN;
  const int ntiles = (N + kBN - 1) / kBN, mt = blockIdx.x / ntiles;   // column tiles first: they share the rows of X
  const int n0 = (blockIdx.x - mt * ntiles) * kBN, m0 = mt * BM;
  const int kb = blockIdx.z * kper, ke = min(K, kb + kper);
  const unsigned sbase = (unsigned)__cvta_generic_to_shared(smem);
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  auto load_a = [&](int st, int k0) {
    const unsigned d = sbase + (unsigned)(st * T::stage) * 4u;
    if (VECA) {
      for (int i = tid; i < BM * (T::BK / 4); i += kGT) {
        const int m = i / (T::BK / 4), k = (i - m * (T::BK / 4)) * 4;
        const bool in = m0 + m < M && k0 + k < ke;
        mma::cp_async16_s(d + (unsigned)(m * T::PA + k) * 4u, in ? X + (size_t)(m0 + m) * K + k0 + k : X, in ? 16 : 0);
      }
    } else {
      for (int i = tid; i < BM * T::BK; i += kGT) {
        const int m = i / T::BK, k = i - m * T::BK;
        const bool in = m0 + m < M && k0 + k < ke;
        mma::cp_async4_s(d + (unsigned)(m * T::PA + k) * 4u, in ? X + (size_t)(m0 + m) * K + k0 + k : X, in ? 4 : 0);
      }
    }
  };
  auto load_b = [&](int st, int k0) {
    const unsigned d = sbase + (unsigned)(st * T::stage + BM * T::PA) * 4u;
    for (int i = tid; i < T::BK * (kBN / 4); i += kGT) {
      const int k = i / (kBN / 4), n = (i - k * (kBN / 4)) * 4;
      const bool in = k0 + k < ke && n0 + n < N;
      mma::cp_async16_s(d + (unsigned)(k * (kBN + 4) + n) * 4u, in ? W + (size_t)(k0 + k) * ldw + n0 + n : W, in ? 16 : 0);
    }
  };
  const ClusterSum shared(smem + T::buf + (LONG ? 16 * T::NT : 0), BM * BN, splits);
  const int steps = ke > kb ? (ke - kb + T::BK - 1) / T::BK : 0;
  for (int s = 0; s < kGStages - 1; ++s)
    if (s < steps) load_a(s, kb + s * T::BK);
  grid_dependency_wait();   // the weight kernel's stores
  for (int s = 0; s < kGStages - 1; ++s) {
    if (s < steps) load_b(s, kb + s * T::BK);
    mma::cp_async_commit();
  }
  for (int s = 0; s < steps; ++s) {
    mma::cp_async_wait<kGStages - 2>();
    __syncthreads();
    const int nx = s + kGStages - 1;
    if (nx < steps) {
      load_a(nx % kGStages, kb + nx * T::BK);
      load_b(nx % kGStages, kb + nx * T::BK);
    }
    mma::cp_async_commit();
    const float* As = smem + (s % kGStages) * T::stage + (ty * 4) * T::PA;
    const float* Bs = smem + (s % kGStages) * T::stage + BM * T::PA + tx * 4;
#pragma unroll
    for (int kk = 0; kk < T::BK / T::KG; kk += 4) {
      const int k = kg * (T::BK / T::KG) + kk;
      float4 a[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(As + i * T::PA + k);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float4 b = *reinterpret_cast<const float4*>(Bs + (k + u) * (kBN + 4));
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float av = u == 0 ? a[i].x : u == 1 ? a[i].y : u == 2 ? a[i].z : a[i].w;
          acc[i][0] = fmaf(av, b.x, acc[i][0]);
          acc[i][1] = fmaf(av, b.y, acc[i][1]);
          acc[i][2] = fmaf(av, b.z, acc[i][2]);
          acc[i][3] = fmaf(av, b.w, acc[i][3]);
        }
      }
    }
    if (LONG && s % T::flush == T::flush - 1 && s + 1 < steps) flush_sums<kGT>(acc, smem + T::buf, tid, s + 1 == T::flush);
  }
  if (LONG && steps > T::flush) add_totals<kGT>(acc, smem + T::buf, tid);
  mma::cp_async_wait<0>();
  // the groups' partial results, then the sum over groups, then over the cluster
  __syncthreads();
  float* red = smem;   // [KG][BM][64]
#pragma unroll
  for (int i = 0; i < 4; ++i)
    *reinterpret_cast<float4*>(red + (kg * BM + ty * 4 + i) * kBN + tx * 4) =
        make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
  __syncthreads();
  const auto out = [&](int i, float v) {
    const int m = m0 + i / kBN, n = n0 + i % kBN;
    if (m < M && n < N) Y[(size_t)m * N + n] = v;
  };
  shared.ready();
  for (int i = tid; i < BM * kBN; i += kGT) {
    float v = red[i];
#pragma unroll
    for (int q = 1; q < T::KG; ++q) v += red[q * BM * kBN + i];
    if (splits > 1) shared.put(i, v);
    else out(i, v);
  }
  if (splits > 1) shared.sum(BM * kBN, tid, kGT, out);
}

// ---- 3 x 3 convolution with W[c][tap][t] -----------------------------------------------------------------------------------
// CTA tile: TT output channels x a TR x TC block of pixels of one image; 4 channels x 4 pixels of a row per thread.  Eight
// input channels per stage; a thread's at most kHaloPer halo positions are the same for every channel, so their offsets
// are worked out once.  The CTAs of a cluster split the input channels.
constexpr int kCC = 8, kHaloPer = 2, kCT = 512;   // channels per stage, halo positions per thread, threads

constexpr int conv_flush(int groups) { return (kChain + 9 * kCC / groups / 2) / (9 * kCC / groups); }   // stages of an accumulator

struct SmallConvGeom {
  int C, T, H, W, ldw, cper, splits;
  int TR, TC, tilesW, tiles, PXQ;   // tile rows / columns (a multiple of 4), pixel quads in use
  int P, CS;                        // halo row pitch, halo floats per channel
  int buf;                          // floats of the stages (and the sum over the groups); the totals follow
  int shared;                       // where the cluster's sum is, behind the totals: the same for all CTAs, whatever share of C they have
  int weight;                       // where the weight is that the CTA forms itself, behind all that
};

// INSIDE: a small weight is formed by each CTA for its channels, in shared memory, instead of by a launch before it: 16 -> 16 channels at
// R = 11, eight 32x32 images, 6.8 -> 6.7 us on the device, and 2 us less for the host, which is what such a call then takes (10.2 -> 8.3 us).
struct ConvWeight {
  KronMode m[4];
  unsigned sdiv[4], fdiv[4];   // 2^32 / ns, nf rounded up (0: 1)
  const float* S;
  int order, R, flip;
};
constexpr int kSP = 12;   // taps of a rank in shared memory: three 16-byte reads

template <int TT, int CG, bool INSIDE>
__global__ void __launch_bounds__(kCT) small_conv_kernel(const SmallConvGeom g, const float* __restrict__ X,
                                                         const float* __restrict__ Wt, float* __restrict__ V,
                                                         const __grid_constant__ ConvWeight f) {
  constexpr int TG = TT / 4;
  constexpr int WS = kCC * 9 * TT;
  extern __shared__ __align__(16) float smem[];
  const int xs = kCC * g.CS, stage = xs + (INSIDE ? 0 : WS);
  const int tid = threadIdx.x, lane = tid & 31;
  const int grp = tid / (kCT / CG), warp = (tid >> 5) % (kCT / CG / 32);   // CG groups of warps share a stage's channels
  // lanes: 8 pixel quads x 4 channel quads; warps: the remaining channel quads first
  const int tq = (lane >> 3) + 4 * (warp % (TG / 4)), pq = (lane & 7) + 8 * (warp / (TG / 4));
  const int n = blockIdx.x / g.tiles, tile = blockIdx.x - n * g.tiles;
  const int h0 = (tile / g.tilesW) * g.TR, w0 = (tile % g.tilesW) * g.TC, t0 = blockIdx.y * TT;
  const int cb = blockIdx.z * g.cper, ce = min(g.C, cb + g.cper);
  const int HW = g.H * g.W;
  const float* Xn = X + (size_t)n * g.C * HW;
  const unsigned sbase = (unsigned)__cvta_generic_to_shared(smem);
  // halo position p -> row p / (TC + 2), column p % (TC + 2); column -1 is stored at index 3 so that pixel 0 is aligned
  int hg[kHaloPer], hs[kHaloPer];
#pragma unroll
  for (int j = 0; j < kHaloPer; ++j) {
    const int p = tid + j * kCT, hr = p / (g.TC + 2), hc = p - hr * (g.TC + 2);
    const int h = h0 + hr - 1, w = w0 + hc - 1;
    hs[j] = hr < g.TR + 2 ? hr * g.P + hc + 3 : -1;
    hg[j] = (hr < g.TR + 2 && h >= 0 && h < g.H && w >= 0 && w < g.W) ? h * g.W + w : -1;
  }
  auto load_x = [&](int st, int c0) {
    const unsigned d = sbase + (unsigned)(st * stage) * 4u;
#pragma unroll
    for (int j = 0; j < kHaloPer; ++j)
      if (hs[j] >= 0) {
#pragma unroll
        for (int c = 0; c < kCC; ++c) {
          const bool in = hg[j] >= 0 && c0 + c < ce;
          mma::cp_async4_s(d + (unsigned)(c * g.CS + hs[j]) * 4u, in ? Xn + (size_t)(c0 + c) * HW + hg[j] : Xn, in ? 4 : 0);
        }
      }
  };
  auto load_w = [&](int st, int c0) {
    const unsigned d = sbase + (unsigned)(st * stage + xs) * 4u;
    for (int i = tid; i < kCC * 9 * (TT / 4); i += kCT) {
      const int row = i / (TT / 4), t = (i - row * (TT / 4)) * 4;
      const bool in = c0 + row / 9 < ce && t0 + t < g.T;
      mma::cp_async16_s(d + (unsigned)(row * TT + t) * 4u, in ? Wt + ((size_t)c0 * 9 + row) * g.ldw + t0 + t : Wt, in ? 16 : 0);
    }
  };
  float acc[4][4];   // [t][px]
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  constexpr int kFlush = conv_flush(CG);
  float* total = smem + g.buf;
  const bool active = pq < g.PXQ;
  const int pr = active ? pq / (g.TC / 4) : 0, pc = active ? (pq - pr * (g.TC / 4)) * 4 : 0;
  const int steps = ce > cb ? (ce - cb + kCC - 1) / kCC : 0;
  const ClusterSum shared(smem + g.shared, TT * g.TR * g.TC, g.splits);
  if (steps > 0) load_x(0, cb);
  float* weight = smem + g.weight;   // [channel][tap][TT], then the taps of the ranks
  if constexpr (INSIDE) {
    mma::cp_async_commit();
    float* taps = weight + g.cper * 9 * TT;
    const float tap = tid < f.R * kSP && tid % kSP < 9 ? f.S[(size_t)(f.flip ? 8 - tid % kSP : tid % kSP) * f.R + tid / kSP] : 0.f;
    // this thread's entry (channel, output): where its factors' values of rank 0 are; four ranks of them, on their way early
    const float* F[4];
    float p[4];
    const int ci = cb + tid / TT, ti = t0 + tid % TT;
    const bool entry = tid < g.cper * TT && ci < ce && ti < g.T;
    if (entry) {
      unsigned s = ci, q = ti;
#pragma unroll
      for (int k = 3; k >= 0; --k) {
        if (k >= f.order) continue;
        const unsigned sn = f.sdiv[k] ? __umulhi(s, f.sdiv[k]) : s, qn = f.fdiv[k] ? __umulhi(q, f.fdiv[k]) : q;
        F[k] = f.m[k].F + (size_t)((s - sn * f.m[k].ns) * f.m[k].fs + (q - qn * f.m[k].nf) * f.m[k].ff) * f.R;
        s = sn;
        q = qn;
      }
    }
    const auto fetch = [&](int r0) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const bool in = r0 + j < f.R;
        p[j] = in ? F[0][r0 + j] : 0.f;
#pragma unroll
        for (int k = 1; k < 4; ++k)
          if (k < f.order && in) p[j] *= F[k][r0 + j];
      }
    };
    if (entry) fetch(0);
    if (tid < f.R * kSP) taps[tid] = tap;
    __syncthreads();
    if (tid < g.cper * TT) {   // at most one entry per thread
      float w[9];
#pragma unroll
      for (int j = 0; j < 9; ++j) w[j] = 0.f;
      if (entry)
        for (int r0 = 0; r0 < f.R; r0 += 4) {
          const float v[4] = {p[0], p[1], p[2], p[3]};
          if (r0 + 4 < f.R) fetch(r0 + 4);
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            if (r0 + u >= f.R) break;
            const float* tr = taps + (r0 + u) * kSP;
            const float4 a = *reinterpret_cast<const float4*>(tr), b = *reinterpret_cast<const float4*>(tr + 4);
            const float x[9] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, tr[8]};
#pragma unroll
            for (int j = 0; j < 9; ++j) w[j] = fmaf(v[u], x[j], w[j]);
          }
        }
#pragma unroll
      for (int j = 0; j < 9; ++j) weight[(tid / TT * 9 + j) * TT + tid % TT] = w[j];
    }
  } else {
    grid_dependency_wait();
    if (steps > 0) load_w(0, cb);
    mma::cp_async_commit();
  }
  for (int s = 0; s < steps; ++s) {
    if (s + 1 < steps) {
      load_x((s + 1) & 1, cb + (s + 1) * kCC);
      if (!INSIDE) load_w((s + 1) & 1, cb + (s + 1) * kCC);
    }
    mma::cp_async_commit();
    mma::cp_async_wait<1>();
    __syncthreads();
    if (active) {
      const float* xb = smem + (s & 1) * stage + pr * g.P + pc + 4;
      const float* wb = (INSIDE ? weight + s * WS : smem + (s & 1) * stage + xs) + tq * 4;
#pragma unroll 2
      for (int cc = 0; cc < kCC / CG; ++cc) {
        const int c = grp * (kCC / CG) + cc;
#pragma unroll
        for (int y = 0; y < 3; ++y) {
          const float* xr = xb + c * g.CS + y * g.P;
          const float4 m = *reinterpret_cast<const float4*>(xr);
          const float x[6] = {xr[-1], m.x, m.y, m.z, m.w, xr[4]};
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            const float4 wv = *reinterpret_cast<const float4*>(wb + (c * 9 + y * 3 + k) * TT);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              acc[0][j] = fmaf(wv.x, x[j + k], acc[0][j]);
              acc[1][j] = fmaf(wv.y, x[j + k], acc[1][j]);
              acc[2][j] = fmaf(wv.z, x[j + k], acc[2][j]);
              acc[3][j] = fmaf(wv.w, x[j + k], acc[3][j]);
            }
          }
        }
      }
    }
    if (s % kFlush == kFlush - 1 && s + 1 < steps) flush_sums<kCT>(acc, total, tid, s + 1 == kFlush);
    __syncthreads();
  }
  if (steps > kFlush) add_totals<kCT>(acc, total, tid);
  float* Vn = V + (size_t)n * g.T * HW;
  const int npx = g.TR * g.TC;
  // the channel groups, then the cluster, are added in shared memory over the stage buffers: [group][t][px] (every
  // thread is past its last read)
  if (active)
#pragma unroll
    for (int i = 0; i < 4; ++i)
      *reinterpret_cast<float4*>(smem + (grp * TT + tq * 4 + i) * npx + pr * g.TC + pc) =
          make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
  __syncthreads();
  const auto out = [&](int i, float v) {
    const int t = t0 + i / npx, px = i % npx, h = h0 + px / g.TC, w = w0 + px % g.TC;
    if (t < g.T && h < g.H && w < g.W) Vn[(size_t)t * HW + h * g.W + w] = v;
  };
  shared.ready();
  for (int i = tid; i < TT * npx; i += kCT) {
    float v = smem[i];
#pragma unroll
    for (int q = 1; q < CG; ++q) v += smem[q * TT * npx + i];
    if (g.splits > 1) shared.put(i, v);
    else out(i, v);
  }
  if (g.splits > 1) shared.sum(TT * npx, tid, kCT, out);
}

// Dynamic shared memory that lets no more CTAs share an SM than the grid needs: CTAs of a programmatic dependent start
// while the kernel before drains and would otherwise be stacked on the SMs that are free first.
// (A GPC of fewer than 16 SMs has room for one cluster of 8 only: with a CTA per SM 15 clusters are resident at once, 16 are not.  128 -> 16
// channels 7x7 at R = 18, images = clusters, a CTA per SM / two: 11 8.0 / 9.3 us, 14 8.2 / 9.5, 15 8.4 / 9.4, 16 11.9 / 9.6.)
bool paired_clusters(long ctas, int cluster) { return cluster == 8 && ctas > 14 * 8; }
size_t spread_smem(size_t need, long ctas, int cluster, const DeviceInfo& di) {
  const long per = std::max<long>((ctas + di.sm_count - 1) / di.sm_count, paired_clusters(ctas, cluster) ? 2 : 1);
  return per > 4 ? need : std::max(need, (size_t)di.smem_optin / per - (per > 1 ? 1024 : 0));
}

// The tallest tile that leaves a CTA for most SMs (tall tiles form fewer half products per entry); a weight too small
// even for 16-row tiles is shared out over the ranks as well.
struct KronPlan {
  int PA, nb, ta, splits, rper;
  long ctas;
};
KronPlan kron_plan(int order, const int* slow, const int* fast, int R, int taps, const DeviceInfo& di) {
  KronPlan p{};
  int PB = 1;
  p.PA = taps;
  for (int k = 0; k < order; ++k) (k < order / 2 ? p.PA : PB) *= slow[k] * fast[k];
  p.nb = ceil_div(PB, kTB);
  p.ta = 64;
  while (p.ta > 16 && (long)p.nb * ceil_div(p.PA, p.ta) * 5 < 4L * di.sm_count) p.ta /= 2;
  const long tiles = (long)p.nb * ceil_div(p.PA, p.ta);
  p.splits = pick_cluster(tiles, R, 16, di.sm_count);
  p.rper = ceil_div(R, p.splits);
  p.ctas = tiles * p.splits;
  return p;
}

struct GemmPlan {
  int bm, bn, splits, kper;
  long tiles;
};
GemmPlan gemm_plan(int M, int N, int K, const DeviceInfo& di) {
  GemmPlan p{};
  // the tallest tile that leaves enough CTAs for one wave once a cluster splits K eight ways
  const auto enough = [&](int bm) { return M > bm / 2 && (long)ceil_div(M, bm) * ceil_div(N, 64) * 8 >= di.sm_count; };
  p.bm = enough(64) ? 64 : enough(32) ? 32 : 16;
  p.bn = p.bm == 16 && (long)ceil_div(M, 16) * ceil_div(N, 64) * 8 < di.sm_count ? 32 : 64;
  const auto tiles = [&] {
    p.tiles = (long)ceil_div(M, p.bm) * ceil_div(N, p.bn);
    p.splits = pick_cluster(p.tiles, K, 64, di.sm_count);
  };
  tiles();
  if (p.bn == 32 && (M <= 8 || p.tiles * 8 < di.sm_count)) {   // half of the rows, unless that is many clusters of 8
    p.bm = 8;
    tiles();
    if (p.splits == 8 && p.tiles > 8) {
      p.bm = 16;
      tiles();
    }
  }
  p.kper = (int)align_up((size_t)ceil_div(K, p.splits), 4);
  return p;
}

// The CTAs form the weight where that is one entry per thread, of at most so many ranks.  Calls one after the other, weight by a launch /
// inside (the launch also costs the host 2 us): 16 -> 10 channels at R = 14 9.2 / 8.3 us, 12 at R = 15 11.9 / 10.3; two entries: 60 channels at
// R = 5 14.4 / 16.4, 192 -> 24 at R = 14 10.3 / 12.3; 28 ranks: 16 -> 12 9.3 / 10.3.
constexpr int kInside = 16;

struct ConvPlan {
  int tt, cgroups;
  long tiles;
  size_t floats, inside;   // of shared memory, without the weight and with it formed inside
  SmallConvGeom g;
};
ConvPlan conv_plan(int N, int C, int T, int H, int W, int R, const DeviceInfo& di) {
  ConvPlan p{};
  SmallConvGeom& g = p.g;
  const int tt = p.tt = T <= 16 ? 16 : T <= 32 ? 32 : 64;
  // two channel groups share the 16 warps; eight (four with 64 output channels: a warp holds 16 of them), with a quarter
  // or half of the pixels per CTA, where there are few pixels
  const bool few = (long)N * ceil_div(H * W, kCT * 2 / (tt / 4)) * ceil_div(T, tt) * 2 <= di.sm_count;
  p.cgroups = few ? (tt == 64 ? 4 : 8) : 2;
  const int quads = kCT / p.cgroups / (tt / 4);      // pixel quads per CTA
  g.C = C; g.T = T; g.H = H; g.W = W; g.ldw = (T + 3) / 4 * 4;
  // columns of the tile: the width that covers the image with the least waste and halo
  int best = 4;
  double best_cost = 1e300;
  for (int tc = 4; tc <= std::min(32, (W + 3) / 4 * 4); tc += 4) {
    const int tr = std::min(quads / (tc / 4), H);
    if (tr < 1 || (tr + 2) * (tc + 2) > kHaloPer * kCT) continue;
    const double cost = (double)ceil_div(W, tc) * ceil_div(H, tr) * (1.0 + 0.1 * (tr + 2.0) * (tc + 2.0) / (tr * tc));
    if (cost < best_cost) { best_cost = cost; best = tc; }
  }
  g.TC = best;
  g.TR = std::min(quads / (g.TC / 4), H);
  g.tilesW = ceil_div(W, g.TC);
  g.tiles = g.tilesW * ceil_div(H, g.TR);
  g.PXQ = g.TR * (g.TC / 4);
  g.P = g.TC + 8;
  g.CS = (int)align_up((size_t)(g.TR + 2) * g.P, 4);
  p.tiles = (long)N * g.tiles * ceil_div(T, tt);
  g.splits = pick_cluster(p.tiles, C, 2 * kCC, di.sm_count);
  g.cper = (int)align_up((size_t)ceil_div(C, g.splits), kCC);
  const int stages = 2 * kCC * g.CS, sums = p.cgroups * tt * g.TR * g.TC;
  const int totals = ceil_div(g.cper, kCC) > conv_flush(p.cgroups) ? 16 * kCT : 0;   // (the last CTA of a cluster may need none)
  const size_t behind = totals + ClusterSum::floats(tt * g.TR * g.TC);
  g.buf = std::max(stages + 2 * kCC * 9 * tt, sums);
  g.shared = g.buf + totals;
  p.floats = g.buf + behind;
  // the weight of the CTA's channels and the ranks' taps
  if (g.cper * tt <= kCT && R <= kInside) {
    const int buf = std::max(stages, sums);
    const size_t weight = align_up(buf + behind, 4), all = weight + (size_t)g.cper * 9 * tt + (size_t)R * kSP;
    if (all * sizeof(float) <= (size_t)di.smem_optin) {
      g.buf = buf;
      g.shared = buf + totals;
      g.weight = (int)weight;
      p.inside = all;
    }
  }
  return p;
}

double waves(long ctas, const DeviceInfo& di) { return (double)((ctas + di.sm_count - 1) / di.sm_count); }

}  // namespace

// Estimated microseconds of the two forms: waves of CTAs times the work of one, and the weight's entries written.  The coefficients are a
// least-squares fit to the first form of these kernels (tiles of 16 and more rows, 4 x 4 values per thread of the weight, cluster sums by
// reads); with the present ones the estimates are 0.84 to 1.18 of the time of eight of ten products (formed inside: 1.05 to 1.45).  They only
// have to choose: over 1000 drawn products (one to four modes of 1-16, up to 8192 features or 1024 channels, batches to 8192 and images to
// 64 x 64, ranks 1-300), each measured in every form that takes it, the choice is 0.6 % behind the best one all together, and 16 products
// run more than 10 % and 2 us behind: 35 samples 3000 -> 1920 at R = 16 84 us on the tensor cores and 55 here, 69 samples 30 -> 30 at R = 1 10.2
// here and 7.2 factored.
double kron_weight_us(int order, const int* idims, const int* odims, int R, int taps, bool transposed) {
  DeviceInfo di;
  if (device_info(&di)) return 1e300;
  const KronPlan p = kron_plan(order, transposed ? odims : idims, transposed ? idims : odims, R, taps, di);
  double slow = taps, fast = 1;
  for (int k = 0; k < order; ++k) {
    slow *= transposed ? odims[k] : idims[k];
    fast *= transposed ? idims[k] : odims[k];
  }
  return 3.05e-6 * slow * std::ceil(fast / 4) * 4 + 4.07e-4 * waves(p.ctas, di) * p.rper * (p.ta + 64);
}

double dense_kron_us(int B, int order, const int* idims, const int* odims, int R, bool transposed) {
  DeviceInfo di;
  if (device_info(&di)) return -1;
  int K = 1, N = 1;
  for (int k = 0; k < order; ++k) {
    K *= transposed ? odims[k] : idims[k];
    N *= transposed ? idims[k] : odims[k];
  }
  const GemmPlan p = gemm_plan(B, N, K, di);
  const double work = waves(p.tiles * p.splits, di) * p.kper * p.bm * p.bn;
  return 5.1 + kron_weight_us(order, idims, odims, R, 1, transposed) +
         (p.bm == 64 ? 7.93e-6 : p.bm == 32 ? 9.39e-6 : 7.69e-6) * work + 1.54e-6 * ((double)B * K + (double)B * N);
}

double rcp_kron_us(int N, int H, int W, int order, const int* cdims, const int* tdims, int R, bool transposed, bool* inside) {
  DeviceInfo di;
  if (device_info(&di)) return -1;
  int C = 1, T = 1;
  for (int k = 0; k < order; ++k) {
    C *= transposed ? tdims[k] : cdims[k];
    T *= transposed ? cdims[k] : tdims[k];
  }
  const ConvPlan p = conv_plan(N, C, T, H, W, R, di);
  const SmallConvGeom& g = p.g;
  *inside = p.inside > 0;
  const int px = kCT / p.cgroups / (p.tt / 4) * 4;
  const double w = waves(p.tiles * g.splits, di) * g.cper;
  return 5.1 + (p.inside ? 0.2 * R : kron_weight_us(order, cdims, tdims, R, 9, transposed)) +
         (p.tt == 64 ? 6.71e-6 : 5.19e-6) * w * 9 * p.tt * px + 8.04e-4 * w * (g.TR + 2) * (g.TC + 2);
}

// Row pitch of the weight: 16-byte rows.
int kron_weight_ld(int fast) { return (fast + 3) / 4 * 4; }

static KronMode kron_mode(const float* F, int idim, int odim, bool transposed) {
  KronMode m{};
  m.F = F;
  m.ns = transposed ? odim : idim;
  m.nf = transposed ? idim : odim;
  m.fs = transposed ? 1 : odim;
  m.ff = transposed ? odim : 1;
  return m;
}

// the modes and halves of a weight with rows of `ld` entries per tap
static int kron_geom(int order, const int* idims, const int* odims, int R, const float* const* F, const float* S, int taps,
                     bool transposed, bool flip, int ld, long* rows, KronGeom* out) {
  KronMode m[4];
  long slow = 1, fast = 1;
  for (int k = 0; k < order; ++k) {
    m[k] = kron_mode(F[k], idims[k], odims[k], transposed);
    slow *= m[k].ns;
    fast *= m[k].nf;
  }
  const int row = S ? taps * ld : ld;
  if (slow * row > 0x7fffffffL) return fail(B200CP_ERR_UNSUPPORTED, "multiplied-out weight too large");
  long os = row, of = 1;
  for (int k = order - 1; k >= 0; --k) {
    m[k].os = (int)os;
    m[k].of = (int)of;
    os *= m[k].ns;
    of *= m[k].nf;
  }
  KronGeom g{};
  g.R = R;
  g.SA = g.FA = g.SB = g.FB = 1;
  const int ha = order / 2;
  if (S) {
    g.A[g.nA++] = KronMode{S, taps, 1, 1, 0, ld, 0};
    g.SA *= taps;
    g.flip = flip ? 1 : 0;
  }
  for (int k = 0; k < ha; ++k) { g.A[g.nA++] = m[k]; g.SA *= m[k].ns; g.FA *= m[k].nf; }
  for (int k = ha; k < order; ++k) { g.B[g.nB++] = m[k]; g.SB *= m[k].ns; g.FB *= m[k].nf; }
  *rows = slow;
  *out = g;
  return B200CP_OK;
}

// W[s][ld] (dense) or W[s][tap][ld] (S given): slow side = inputs, or outputs with `transposed`; with `flip` the taps run
// backwards (a data gradient)
int kron_weight_launch(int order, const int* idims, const int* odims, int R, const float* const* F, const float* S,
                       int taps, bool transposed, bool flip, float* W, cudaStream_t st, bool stacked) {
  long fast = 1, rows;
  for (int k = 0; k < order; ++k) fast *= transposed ? idims[k] : odims[k];
  KronGeom g;
  if (int rc = kron_geom(order, idims, odims, R, F, S, taps, transposed, flip, kron_weight_ld((int)fast), &rows, &g)) return rc;
  DeviceInfo di;
  if (int rc = device_info(&di)) return rc;
  const KronPlan p = kron_plan(order, transposed ? odims : idims, transposed ? idims : odims, R, S ? taps : 1, di);
  const int ta = p.ta, splits = p.splits;
  g.rper = p.rper;
  // (two CTAs of the product to an SM, beside this grid's, would all be placed as pairs: 160 -> 192 channels 10x10 at R = 28 16.7 us, later 12.8)
  g.early = p.ctas <= (stacked ? di.sm_count / 2 : di.sm_count);
  const dim3 grid(p.nb, ceil_div(p.PA, ta), splits);
#define KRON_T(TAV, TAPV)                                                                                               \
  do {                                                                                                                  \
    if constexpr (kron_smem<TAV>() > 44 * 1024) {   /* (48 KB with the offsets need no limit raised) */                  \
      static std::atomic<int> set[64];                                                                                  \
      B200CP_CUDA_OK(ensure_dynamic_smem(reinterpret_cast<const void*>(kron_weight_kernel<TAV, TAPV>), set, (int)kron_smem<TAV>())); \
    }                                                                                                                   \
    B200CP_CUDA_OK(launch_cluster(kron_weight_kernel<TAV, TAPV>, grid, dim3(kKT), kron_smem<TAV>(), st, splits, false, g, W)); \
  } while (0)
#define KRON(TAV)                                                                                                       \
  do {                                                                                                                  \
    if (S) KRON_T(TAV, true);                                                                                           \
    else KRON_T(TAV, false);                                                                                            \
  } while (0)
  if (ta == 64) KRON(64);
  else if (ta == 32) KRON(32);
  else KRON(16);
#undef KRON
#undef KRON_T
  B200CP_LAUNCH_OK("kron_weight_kernel");
  return B200CP_OK;
}

// Large weights, whose 128 x 128 tiles fill the GPU: 4096 x 4096 at R = 32 42 us with the exponents, against 86 for the fp32 weight and
// its split; but 1000 x 1000 at R = 16 21 against 13, 4096 x 64 at R = 64 50 against 20.
bool kron_planes_takes(int order, const int* idims, const int* odims, int R, int sm_count) {
  double pa = 1, pb = 1;
  for (int k = 0; k < order; ++k) (k < order / 2 ? pa : pb) *= (double)idims[k] * odims[k];
  return R <= kKeep && std::ceil(pa / kPT) * std::ceil(pb / kPT) >= 2.0 * sm_count && pa >= kPT && pb >= kPT;
}

// The same weight as hi / lo planes of `plane` values with rows of ldo, a multiple of 4, and one exponent per row (kron_planes_takes).
int kron_planes_launch(int order, const int* idims, const int* odims, int R, const float* const* F, bool transposed, int ldo,
                       void* hi, size_t plane, int* ex, cudaStream_t st) {
  KronGeom g;
  long rows;
  if (int rc = kron_geom(order, idims, odims, R, F, nullptr, 1, transposed, false, ldo, &rows, &g)) return rc;
  DeviceInfo di;
  if (int rc = device_info(&di)) return rc;
  if (R > kKeep) return fail(B200CP_ERR_UNSUPPORTED, "multiplied-out weight: rank %d", R);
  size_t table = 0;
  for (int k = 0; k < order; ++k) table += sizeof(float) * kron_mode_of(g, k).ns * R;
  static std::atomic<int> exset[64];
  B200CP_CUDA_OK(ensure_dynamic_smem(reinterpret_cast<const void*>(kron_exponent_kernel), exset, (int)table));
  kron_exponent_kernel<<<(unsigned)((rows + kRowsEx - 1) / kRowsEx), 32 * kRowsEx, table, st>>>(g, (int)rows, ex);
  B200CP_LAUNCH_OK("kron_exponent_kernel");
  const int atiles = ceil_div(g.SA * g.FA, kPT), btiles = ceil_div(g.SB * g.FB, kPT);
  if (atiles > 65535) return fail(B200CP_ERR_UNSUPPORTED, "multiplied-out weight too large");
  static std::atomic<int> set[2][64];
  const auto kernel = R > 64 ? kron_planes_kernel<true> : kron_planes_kernel<false>;
  B200CP_CUDA_OK(ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), set[R > 64], (int)kPlanesSmem));
  // as many CTAs as are resident at once share the tiles of B
  const int walkers = std::min(btiles, std::max(1, 2 * di.sm_count / atiles));
  const dim3 grid(walkers, atiles);
  const bool vec = !(ldo & 7) && !(plane & 7) && !(reinterpret_cast<uintptr_t>(hi) & 15);
  B200CP_CUDA_OK(launch_kernel(kernel, grid, dim3(256), kPlanesSmem, st, true, g, ldo, btiles, ex, static_cast<__half*>(hi), plane, vec));
  B200CP_LAUNCH_OK("kron_planes_kernel");
  return B200CP_OK;
}

// Reads (and clears) the status word; the caller has synchronised the device.
int kron_device_status(int* out) {
  int v = 0, zero = 0;
  B200CP_CUDA_OK(cudaMemcpyFromSymbol(&v, g_kron_status, sizeof(int)));
  if (v) B200CP_CUDA_OK(cudaMemcpyToSymbol(g_kron_status, &zero, sizeof(int)));
  *out = v;
  return B200CP_OK;
}

int small_gemm_launch(int M, int N, int K, const float* X, const float* W, float* Y, cudaStream_t st) {
  DeviceInfo di;
  if (int rc = device_info(&di)) return rc;
  const int ldw = kron_weight_ld(N);
  const bool vec = !(K & 3) && !(reinterpret_cast<uintptr_t>(X) & 15);
  const GemmPlan p = gemm_plan(M, N, K, di);
  const int bm = p.bm, bn = p.bn, splits = p.splits, kper = p.kper;
  const long tiles = p.tiles;
  if (tiles > 0x7fffffffL || M > 0x7fffffff - 64) return fail(B200CP_ERR_UNSUPPORTED, "dense: batch of %d rows too large", M);
  const dim3 grid((unsigned)tiles, 1, splits);   // (grid y would end at 65535 row tiles)
#define SMALL_GEMM_L(BMV, BNV, V, L)                                                                                    \
  do {                                                                                                                  \
    static std::atomic<int> set[64];                                                                                    \
    const size_t smem = spread_smem(GemmTile<BMV, BNV>::smem(kper), tiles * splits, splits, di);                                \
    B200CP_CUDA_OK(ensure_dynamic_smem(reinterpret_cast<const void*>(small_gemm_kernel<BMV, BNV, V, L>), set, di.smem_optin)); \
    B200CP_CUDA_OK(launch_cluster(small_gemm_kernel<BMV, BNV, V, L>, grid, dim3(GemmTile<BMV, BNV>::NT), smem, st, splits, true, \
                                  X, W, Y, M, N, K, ldw, kper, splits));                                                \
  } while (0)
#define SMALL_GEMM(BMV, BNV, V)                                                                                         \
  do {                                                                                                                  \
    if (GemmTile<BMV, BNV>::is_long(kper)) SMALL_GEMM_L(BMV, BNV, V, true);                                             \
    else SMALL_GEMM_L(BMV, BNV, V, false);                                                                              \
  } while (0)
  if (bm == 8) { if (vec) SMALL_GEMM(8, 32, true); else SMALL_GEMM(8, 32, false); }
  else if (bn == 32) { if (vec) SMALL_GEMM(16, 32, true); else SMALL_GEMM(16, 32, false); }
  else if (bm == 16) { if (vec) SMALL_GEMM(16, 64, true); else SMALL_GEMM(16, 64, false); }
  else if (bm == 32) { if (vec) SMALL_GEMM(32, 64, true); else SMALL_GEMM(32, 64, false); }
  else { if (vec) SMALL_GEMM(64, 64, true); else SMALL_GEMM(64, 64, false); }
#undef SMALL_GEMM_L
#undef SMALL_GEMM
  B200CP_LAUNCH_OK("small_gemm_kernel");
  return B200CP_OK;
}

// how a cluster shares out the channels: its CTAs, stages of the first and of the last, stages after which an accumulator is added up
int conv_shares(int N, int C, int T, int H, int W, int R, int* out) {
  DeviceInfo di;
  if (int rc = device_info(&di)) return rc;
  const ConvPlan p = conv_plan(N, C, T, H, W, R, di);
  out[0] = p.g.splits;
  out[1] = ceil_div(std::min(C, p.g.cper), kCC);
  out[2] = ceil_div(std::max(0, C - (p.g.splits - 1) * p.g.cper), kCC);
  out[3] = conv_flush(p.cgroups);
  return B200CP_OK;
}

// V = W * X, the weight multiplied out to Wt, or (Wt null) formed inside
int small_conv_launch(int N, int H, int W, int order, const int* cdims, const int* tdims, int R, const float* const* A, const float* S,
                      bool transposed, const float* X, float* Wt, float* V, cudaStream_t st) {
  DeviceInfo di;
  if (int rc = device_info(&di)) return rc;
  int C = 1, T = 1;
  ConvWeight f{};
  f.order = order; f.R = R; f.S = S; f.flip = transposed;
  for (int k = 0; k < order; ++k) {
    f.m[k] = kron_mode(A[k], cdims[k], tdims[k], transposed);
    f.sdiv[k] = f.m[k].ns > 1 ? (unsigned)((0x100000000ull + f.m[k].ns - 1) / f.m[k].ns) : 0;
    f.fdiv[k] = f.m[k].nf > 1 ? (unsigned)((0x100000000ull + f.m[k].nf - 1) / f.m[k].nf) : 0;
    C *= f.m[k].ns;
    T *= f.m[k].nf;
  }
  const ConvPlan p = conv_plan(N, C, T, H, W, Wt ? INT_MAX : R, di);
  const SmallConvGeom& g = p.g;
  const int tt = p.tt, cgroups = p.cgroups;
  const long tiles = p.tiles;
  const size_t smem = sizeof(float) * (Wt ? p.floats : p.inside);
  dim3 grid((unsigned)(N * g.tiles), ceil_div(T, tt), g.splits);
  if ((long)N * g.tiles > 0x7fffffffL) return fail(B200CP_ERR_UNSUPPORTED, "rcp: too many tiles");
  if (Wt)
    if (int rc = kron_weight_launch(order, cdims, tdims, R, A, S, 9, transposed, transposed, Wt, st, paired_clusters(tiles * g.splits, g.splits)))
      return rc;
#define SMALL_CONV_I(TTV, CGV, IN)                                                                                        \
  do {                                                                                                                \
    static std::atomic<int> set[64];                                                                                  \
    const auto kernel = small_conv_kernel<TTV, CGV, IN>;                                                              \
    B200CP_CUDA_OK(ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), set, di.smem_optin));                   \
    B200CP_CUDA_OK(launch_cluster(kernel, grid, dim3(kCT), IN ? smem : spread_smem(smem, tiles * g.splits, g.splits, di), st, \
                                  g.splits, !IN, g, X, Wt, V, f));                                                    \
  } while (0)
#define SMALL_CONV(TTV, CGV)                                                                                              \
  do {                                                                                                                \
    if (Wt) SMALL_CONV_I(TTV, CGV, false);                                                                            \
    else SMALL_CONV_I(TTV, CGV, true);                                                                                \
  } while (0)
  if (cgroups == 2) {
    if (tt == 16) SMALL_CONV(16, 2);
    else if (tt == 32) SMALL_CONV(32, 2);
    else SMALL_CONV(64, 2);
  } else {
    if (tt == 16) SMALL_CONV(16, 8);
    else if (tt == 32) SMALL_CONV(32, 8);
    else SMALL_CONV(64, 4);
  }
#undef SMALL_CONV
#undef SMALL_CONV_I
  B200CP_LAUNCH_OK("small_conv_kernel");
  return B200CP_OK;
}

}  // namespace b200cp
