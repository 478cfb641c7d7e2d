// D[m][n] = sum_k A[m][k] B[n][k] on the tcgen05 tensor cores with the accuracy of fp32 sums: the gradient product of the
// CP dense layer and of the reshaped-CP convolution, and the product of either layer with its multiplied-out weight.
//
// Accuracy, products with the weight.  A value x is scaled by a power of two (exact) so that the largest of its row is in
// [2^14, 2^15), and split into hi = fp16(x), lo = fp16(x - hi): 22 bits, down to 2^-18 of the row's largest value; smaller values
// have an absolute error of 2^-40 of it.  The product is hi*hi + hi*lo + lo*hi (three tcgen05.mma.kind::f16; a tf32 split has
// the same 22 bits at half the rate).
// Gradient products.  The sum runs over samples (pixels) there, and one of them may be any number of binades above the others and
// still add nothing (a masked sample: its gradient is zero).  No exponent that samples share keeps the others exact, so each
// value keeps its own: x is the sum of three bf16 values, 24 bits, and the product six of theirs (without those below 2^-24).
// Twice the tensor work: 4096 x 4096 x 4096 637 us, nine taps of 256 x 256 at 32 x 28 x 28 153, where fp16 pairs with
// an exponent per column took 326 and 84 and lost all others beside one sample of 1e12.  (Pairs only where all of a column's values lie
// within 29 binades, 318 and 77, still hold 23 of the 24 bits: a value in four is one unit off, and 2049 x 2049 is not exact.)
// The tensor core cuts its fp32 sums off instead of rounding them, which over thousands of terms is a bias of 1e-5 (4096
// terms in one accumulator: 2.9e-5 against float64 in the factor gradients).  So an accumulator holds 64 or 32 terms, the small
// products first, and is then added to a total in registers, in fp32 with rounding.
//
// Layout.  A pair of CTAs (cta_group::2) forms a 256 x BN tile: each loads its 128 rows of A and half of the columns of B,
// 64 KB a step for 3 x 128 x 256 x 64 multiply-adds (gradients: 48 KB for 6 x 128 x 256 x 32).  With one CTA per 128 x 256 tile
// it would be 96 KB, and the stream from L2 is what bounds such a kernel.  TMA fills a ring of three to five stages, one thread
// of the pair issues the products into two (narrower tiles: four) accumulators in turn, and the other warps of each CTA move the
// finished ones to the totals meanwhile (the totals are half of the register file: that is what ends the tile at 128 x 256 per CTA).
// The pairs are persistent: the totals of a tile are stored while the products of the next have begun.
// Operands: K-major ([row][k], 64 k = one 128-byte swizzled row) or MN-major ([k][row], boxes of 64 rows), both taken by
// tcgen05 directly, so that neither the batch-major activations of a gradient nor the weight are transposed in memory.
// Measured, 4096 x 4096 x 4096 with the weight: 305 to 335 us = 1.35 to 1.23 PFLOP/s of fp16 products, and 1.29 of bf16 products in
// the gradient, where cuBLAS sustains 1.40 under the power cap.  Without the cut of the last round of tiles 348 us; with eight
// read-out warps of 128 columns instead of sixteen 317 against 307.
// Roles (TMA warp, MMA warp, read-out warps) meet only through mbarriers; every wait is bounded, and a wait that
// runs out sets a status word and lets the CTA leave through its normal exit (TMEM released).
#include <algorithm>
#include <cfloat>
#include <cstdio>
#include <cstdlib>

#include "common.cuh"
#include "tc_common.cuh"

namespace b200cp {

__device__ int g_gemm_tc_status = 0;  // 0 ok; otherwise (code << 16) | (linear block index & 0xffff)

namespace {

using namespace tc;

constexpr int kBM = 256;              // rows of a pair's tile: 128 per CTA
constexpr int kKS = 64, kGradKS = 32; // K of one step, K-major and MN-major

template <int BN, bool MN>
struct Tile {
  static constexpr int ks = MN ? kGradKS : kKS, planes = MN ? 3 : 2;
  static constexpr int box = planes * ks * 128;                         // MN-major: 64 rows, all planes
  static constexpr int aplane = MN ? ks * 128 : 128 * 128, bplane = MN ? ks * 128 : BN / 2 * 128;   // from one plane to the next
  static constexpr int abytes = planes * 128 * ks * 2;
  static constexpr int stage = abytes + planes * BN / 2 * ks * 2;       // 64, 48, 40 KB; MN-major: 48, 36 KB
  static constexpr int stages = MN ? (BN == 256 ? 4 : 5) : BN == 256 ? 3 : BN == 128 ? 4 : 5;
  static constexpr int depth = BN == 256 ? 2 : 4;                       // accumulators
  static constexpr int tmem_cols = depth * BN;                          // 512, 512, 256
  static constexpr int cols = BN == 64 ? 32 : 64;                       // of a read-out warp
  static constexpr int readers = 4 * BN / cols;                         // read-out warps: 16, 8, 8
  static constexpr int threads = 64 + 32 * readers;                     // warp 0 TMA, warp 1 MMA, the others read-out
  static constexpr size_t smem = (size_t)stages * stage + 1024 + 256;
};

struct SplitGemm {
  int M, N;
  int tiles_m, tiles_n;          // tiles of one result (a weight gradient has one result per tap)
  // Work units in the order in which the pairs take them: `whole` tiles with all K steps, as many as fill the pairs an
  // integer number of times, then the tiles left over, each cut into `splits` ranges of `steps` K steps.
  int whole, units, splits, steps, total;
  int group;                     // K of an accumulator, in instructions of 16 (see kShortSum)
  int kc, Kc;                    // K-major: steps and channels per tap (dense: one tap); MN-major: Kc = rows of K
  int FW, padH, padW, Wp;        // a filter tap (y, x) shifts the rows of A by (y - padH) * Wp + (x - padW)
  // K-major: a value of A stands for 2^ea of itself, one of B for 2^eb.  Rows of A with one exponent over all of K: added at the end.
  // In a convolution the row that a step reads moves with the tap, so the totals take 2^(ea - 24) of each step and
  // 2^(eb + 24) at the end: 24 binades for sums of values near the largest float.
  const int *ea, *eb;
  float* out;                    // entry (m, n) of result p at out + p * result + off(m) + n * ldn
  size_t result;
  float* partial;                // [unit - whole][BN][256] sums of the cut tiles, without the exponents
  long ldm, ldn;                 // off(m) = m * ldm, or, for the pixels of a convolution:
  int vec;                       // ldn == 1 and 16-byte rows
  int H, W, PP;                  // rows are n * PP + h * Wp + w; off = (n * N * H + h) * W + w, ring pixels have none
  // Gradient of a filter with a ring: the images [n][M][H][W] and [n][N][H][W], and a word per 32 pixels of each (see edge_pixels)
  const float *x, *dv;
  const int* dropped;
};

// ---- PTX of a CTA pair --------------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// the same shared variable in the leader CTA of the pair
__device__ __forceinline__ uint32_t leader_addr(uint32_t p) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(p), "r"(0));
  return r;
}
__device__ __forceinline__ void arrive_cluster(uint32_t addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// into this CTA's shared memory, counted on a barrier of either CTA of the pair (no multicast)
__device__ __forceinline__ void tma_load_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], "
      "[%2];" ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z), "r"(0)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(ncols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void mma_f16_pair(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)accumulate)
      : "memory");
}
// one arrival on the barrier of both CTAs when the products issued so far have completed
__device__ __forceinline__ void commit_pair(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
      "h"((uint16_t)3)
      : "memory");
}
// registers -> TMEM: 16 columns of the warp's lane quarter
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const float* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};" ::"f"(v[0]),
      "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "f"(v[8]), "f"(v[9]), "f"(v[10]),
      "f"(v[11]), "f"(v[12]), "f"(v[13]), "f"(v[14]), "f"(v[15]), "r"(taddr)
      : "memory");
}

// Instruction descriptor for kind::f16 with fp32 accumulation, M = 256 (a pair).
// MN-major operands are bf16.
__host__ __device__ constexpr uint32_t make_idesc_f16(uint32_t n, uint32_t mn) {
  return (1u << 4) | (mn << 7) | (mn << 10) | (mn << 15) | (mn << 16) | ((n >> 3) << 17) | ((256u >> 4) << 24);
}

// Bounded wait shared by the roles: gives up after about a second, or as soon as another role of the CTA has given up.
// (Shared-memory addresses in 32 bits: the read-out warps have no register to spare.)
__device__ __forceinline__ bool wait_or_abort(uint32_t bar, uint32_t parity, uint32_t abort_flag) {
  long long t0 = 0;
  for (int it = 0;; ++it) {
    uint32_t done;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
    if ((it & 31) == 31) {
      uint32_t given_up;
      asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(given_up) : "r"(abort_flag) : "memory");
      if (given_up) return false;
      if (t0 == 0) t0 = clock64();
      if (clock64() - t0 > 1500000000ll) {
        asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(abort_flag), "r"(1) : "memory");
        return false;
      }
    }
  }
}

__device__ __forceinline__ int tap_shift(const SplitGemm& g, int tap);
struct UnitAt {
  int m0, n0, tap, shift, first, nsteps;   // tap of the result; shift: of the rows of A (MN-major), by that tap
};
template <int BN, bool MN>
__device__ __forceinline__ UnitAt unit_at(const SplitGemm& g, int unit) {
  UnitAt t;
  const int v = unit - g.whole, tile = v < 0 ? unit : g.whole + v / g.splits;
  const int per = g.tiles_m * g.tiles_n, r = tile % per;
  t.tap = tile / per;
  t.n0 = (r / g.tiles_m) * BN;
  t.m0 = (r % g.tiles_m) * kBM;
  t.shift = MN ? tap_shift(g, t.tap) : 0;
  t.first = v < 0 ? 0 : (v % g.splits) * g.steps;
  t.nsteps = v < 0 ? g.total : min(g.steps, g.total - t.first);
  return t;
}
// Where a step of a unit is in K: its tap (of the sum over taps of a convolution) and its place in the tap.
struct StepAt {
  int tap, c;
};
template <bool CONV>
__device__ __forceinline__ StepAt step_at(const SplitGemm& g, int k) {
  const int tap = CONV ? k / g.kc : 0;
  return StepAt{tap, k - tap * g.kc * (CONV ? 1 : 0)};
}
template <bool CONV>
__device__ __forceinline__ void next_step(const SplitGemm& g, StepAt& k) {
  if (++k.c == g.kc && CONV) {
    k.c = 0;
    ++k.tap;
  }
}
// instructions of 16 k of a step
template <int KS>
__device__ __forceinline__ int k16_of(const SplitGemm& g, int c) {
  const int left = g.Kc - c * KS;
  return left >= KS ? KS / 16 : (left + 15) / 16;
}
__device__ __forceinline__ int tap_shift(const SplitGemm& g, int tap) {
  const int y = tap / g.FW;
  return (y - g.padH) * g.Wp + (tap - y * g.FW - g.padW);
}
// where row m of a result begins, and whether it has one (a convolution's ring pixels have none)
template <bool CONV>
__device__ __forceinline__ bool row_at(const SplitGemm& g, int m, long* off) {
  bool in = m < g.M;
  *off = (long)m * g.ldm;
  if (CONV) {
    const int n = m / g.PP, p = m - n * g.PP, h = p / g.Wp, w = p - h * g.Wp;
    in = in && h < g.H && w < g.W;
    *off = ((long)n * g.N * g.H + h) * g.W + w;
  }
  return in;
}

// A pixel of the ring is zero, and one at the edge of an image that is not finite would make NaN of it, in the taps that reach beside the image
// there.  So split_pixels_kernel takes such pixels for zero and says which 32 (a step) hold one, and here those of a unit's steps make NaN of the sums
// that do meet them (as the products of their parts would): a read-out warp for its own rows and columns.  Finite images pay for a look at a
// word per step; in 32 of 256 channels 28x28 a corner of one, of all channels, costs 13 us, and a row of every image 67.
template <int BN>
__device__ __noinline__ void edge_pixels(const SplitGemm& g, int unit) {
  constexpr int count = Tile<BN, true>::cols;
  const UnitAt u = unit_at<BN, true>(g, unit);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c0 = ((warp - 2) >> 2) * count, HW = g.H * g.W, padH = g.padH, padW = g.padW;
  const int in_tile = (int)cluster_rank() * 128 + (warp & 3) * 32 + lane, m = u.m0 + in_tile, n0 = u.n0 + c0;
  const bool cut = unit >= g.whole && g.splits > 1;
  const long ldn = cut ? kBM : g.ldn;
  float* dst = cut ? g.partial + ((size_t)(unit - g.whole) * BN + c0) * kBM + in_tile : g.out + u.tap * g.result + m + n0 * ldn;   // (ldm is 1)
  const int y = u.tap / g.FW - padH, x = u.tap % g.FW - padW, steps = (g.Kc + kGradKS - 1) / kGradKS, end = u.first + u.nsteps;
  bool row = false;
#pragma unroll 8
  for (int c = 0; c < count; ++c) row |= m < g.M && n0 + c < g.N && dst[c * ldn] == dst[c * ldn];
  if (!__any_sync(0xffffffffu, row)) return;   // NaN already: whole images of it
  row = false;
  uint64_t cols = 0;
#pragma unroll 1
  for (int grad = 0; grad < 2; ++grad) {
    const int dy = grad ? y : -y, dx = grad ? x : -x;   // a pixel of x at (h, w) is met by one of dv at (h - y, w - x)
    for (int k0 = u.first; k0 < end; k0 += 32)
      for (unsigned todo = __ballot_sync(0xffffffffu, k0 + lane < end && g.dropped[grad * steps + min(k0 + lane, end - 1)]); todo; todo &= todo - 1) {
        const int first = (k0 + __ffs(todo) - 1) * kGradKS;
#pragma unroll 4
        for (int i = 0; i < kGradKS; ++i) {
          const int n = (first + i) / g.PP, q = first + i - n * g.PP, h = q / g.Wp, w = q - h * g.Wp;
          if (first + i >= g.Kc || h >= g.H || w >= g.W || h + dy < 0 || h + dy >= g.H || w + dx < 0 || w + dx >= g.W) continue;
          if (h >= padH && h < g.H - padH && w >= padW && w < g.W - padW) continue;
          const size_t at = (size_t)h * g.W + w;
          if (!grad) {
            row = row || (m < g.M && abs_bits(g.x[((size_t)n * g.M + m) * HW + at]) >= 0x7f800000u);
          } else {
            for (int c = 0; c < count; c += 32) {
              const bool in = c + lane < count && n0 + c + lane < g.N;
              cols |= (uint64_t)__ballot_sync(0xffffffffu, in && abs_bits(g.dv[((size_t)n * g.N + (in ? n0 + c + lane : 0)) * HW + at]) >= 0x7f800000u) << c;
            }
          }
        }
      }
  }
  if (m >= g.M) return;
  for (int c = 0; c < count && n0 + c < g.N; ++c)
    if (row || (cols >> c & 1)) dst[c * ldn] = __int_as_float(0x7fffffff);
}

template <int BN, bool MN, bool CONV>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(Tile<BN, MN>::threads, 1)
split_gemm_kernel(const __grid_constant__ SplitGemm g, const __grid_constant__ CUtensorMap mapA,
                  const __grid_constant__ CUtensorMap mapB) {
  using T = Tile<BN, MN>;
  constexpr int kStages = T::stages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + kStages * T::stage);
  uint64_t* full = bars;                 // [kStages] the leader's: the stage of both CTAs has landed  (tx bytes)
  uint64_t* empty = full + kStages;      // [kStages] the products that read the stage are done         (commit, both CTAs)
  uint64_t* accfull = empty + kStages;   // [depth] the accumulator is complete                         (commit, both CTAs)
  uint64_t* accfree = accfull + 4;       // [depth] the leader's: read out by the warps of both CTAs
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accfree + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* edges = abort_flag + 1;   // pixels at the edges were taken for zero

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = (int)cluster_rank(), pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;

  if (tid == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < T::depth; ++i) {
      mbar_init(&accfull[i], 1);
      mbar_init(&accfree[i], 2 * T::readers);
    }
    *abort_flag = 0;
    *edges = 0;
    fence_barrier_init();
    tma_prefetch_desc(&mapA);
    tma_prefetch_desc(&mapB);
  }
  if (warp == 1) tmem_alloc_pair(tmem_slot, T::tmem_cols);
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t fullb = smem_u32(full), emptyb = smem_u32(empty), accfullb = smem_u32(accfull), accfreeb = smem_u32(accfree),
                 abortb = smem_u32(const_cast<int*>(abort_flag));
  grid_dependency_wait();   // the operand planes

  if (warp == 0) {
    // ================= TMA producer: this CTA's rows of A and its half of the columns of B ==================================
    if (lane == 0) {
      int it = 0;
      bool ok = true;
      for (int unit = pair; unit < g.units && ok; unit += npairs) {
        const UnitAt t = unit_at<BN, MN>(g, unit);
        StepAt k = step_at<CONV>(g, t.first);
        for (int s = 0; s < t.nsteps; ++s, ++it, next_step<CONV>(g, k)) {
          const int slot = it % kStages;
          if (it >= kStages && !(ok = wait_or_abort(emptyb + slot * 8, ((it / kStages) - 1) & 1, abortb))) break;
          if (rank == 0) mbar_expect_tx(&full[slot], 2 * T::stage);
          const uint32_t bar = leader_addr(fullb + slot * 8);
          const uint32_t a = smem_u32(sm) + slot * T::stage, b = a + T::abytes;
          if (MN) {   // boxes of 64 rows x 32 k, all planes; rows of K outside the tensor read as zero
#pragma unroll
            for (int q = 0; q < 2; ++q)
              tma_load_pair(a + q * T::box, &mapA, bar, t.m0 + rank * 128 + q * 64, k.c * T::ks + t.shift, 0);
#pragma unroll
            for (int q = 0; q < BN / 128; ++q)
              tma_load_pair(b + q * T::box, &mapB, bar, t.n0 + rank * (BN / 2) + q * 64, k.c * T::ks, 0);
          } else {    // boxes of 64 k x the rows, both planes; channels past Kc read as zero
            const int shift = CONV ? tap_shift(g, k.tap) : 0;
            tma_load_pair(a, &mapA, bar, k.c * kKS, 0, t.m0 + rank * 128 + shift);
            tma_load_pair(b, &mapB, bar, k.c * kKS, k.tap, t.n0 + rank * (BN / 2));
          }
        }
      }
    }
  } else if (warp == 1) {
    // ================= MMA issuer: one thread of the pair ====================================================================
    if (rank == 0 && lane == 0) {
      const uint32_t idesc = make_idesc_f16(BN, MN ? 1 : 0);
      // K-major: rows of 128 bytes, 8 rows per swizzle atom (SBO 1024); 16 k = 32 bytes on.
      // MN-major: 64 rows of the operand (128 bytes) per k, 8 k per atom (SBO 1024), the next 64 rows LBO on; 16 k = 2048 bytes on.
      const uint64_t d0 = make_smem_desc(0, MN ? T::box : 16, 1024, kSwizzle128B);
      constexpr uint32_t kstep = MN ? 2048 : 32;
      const uint32_t base = smem_u32(sm);
      int it = 0, gi = 0;   // steps, accumulators
      bool ok = true;
      for (int unit = pair; unit < g.units && ok; unit += npairs) {
        const UnitAt t = unit_at<BN, MN>(g, unit);
        StepAt k = step_at<CONV>(g, t.first);
        for (int s = 0; s < t.nsteps && ok; ++s, ++it, next_step<CONV>(g, k)) {
          const int slot = it % kStages, kk = k16_of<T::ks>(g, k.c);
          if (!(ok = wait_or_abort(fullb + slot * 8, (it / kStages) & 1, abortb))) break;
          tc_fence_after_sync();
          const uint32_t a = base + slot * T::stage, b = a + T::abytes;
          const uint64_t ah = d0 + (a >> 4), bh = d0 + (b >> 4);
          constexpr uint64_t A1 = T::aplane >> 4, B1 = T::bplane >> 4, A2 = 2 * A1, B2 = 2 * B1;   // to the further planes
          for (int i0 = 0; i0 < kk; i0 += g.group, ++gi) {
            const int buf = gi % T::depth, i1 = min(kk, i0 + g.group);
            if (gi >= T::depth && !(ok = wait_or_abort(accfreeb + buf * 8, (gi / T::depth - 1) & 1, abortb))) break;
            tc_fence_after_sync();
            const uint32_t d = tmem_base + buf * BN;
            if (MN) {   // products of 2^-16 first
              for (int i = i0; i < i1; ++i) {
                const uint64_t o = (uint64_t)((i * kstep) >> 4);
                mma_f16_pair(d, ah + A2 + o, bh + o, idesc, i > i0);
                mma_f16_pair(d, ah + o, bh + B2 + o, idesc, true);
                mma_f16_pair(d, ah + A1 + o, bh + B1 + o, idesc, true);
              }
            }
            for (int i = i0; i < i1; ++i) {
              const uint64_t o = (uint64_t)((i * kstep) >> 4);
              mma_f16_pair(d, ah + A1 + o, bh + o, idesc, MN || i > i0);
              mma_f16_pair(d, ah + o, bh + B1 + o, idesc, true);
            }
            for (int i = i0; i < i1; ++i) {
              const uint64_t o = (uint64_t)((i * kstep) >> 4);
              mma_f16_pair(d, ah + o, bh + o, idesc, true);
            }
            commit_pair(accfullb + buf * 8);
          }
          if (!ok) break;
          commit_pair(emptyb + slot * 8);
        }
      }
    }
  } else {
    // ================= read-out: accumulators -> totals -> global =============================================================
    constexpr int NC = T::cols;
    const int qd = warp & 3, c0 = ((warp - 2) >> 2) * NC;   // the TMEM lane quarter this warp may read, and its columns
    const uint32_t taddr = tmem_base + ((uint32_t)(qd * 32) << 16) + c0;
    if (MN && g.dropped) {   // while the first stages are on their way
      int any = 0;
      for (int i = tid - 64, end = 2 * ((g.Kc + kGradKS - 1) / kGradKS); i < end; i += 32 * T::readers) any |= g.dropped[i];
      if (any) *edges = 1;
      asm volatile("bar.sync 1, %0;" ::"n"(32 * T::readers) : "memory");
    }
    int gi = 0;
    bool ok = true;
    for (int unit = pair; unit < g.units && ok; unit += npairs) {
      float tot[NC];
#pragma unroll
      for (int j = 0; j < NC; ++j) tot[j] = 0.f;
      int buf = 0;
      {
        const UnitAt t = unit_at<BN, MN>(g, unit);
        StepAt k = step_at<CONV>(g, t.first);
        for (int left = t.nsteps; left > 0 && ok; --left, next_step<CONV>(g, k)) {
          float f = 0.f;
          if (CONV) {
            const int px = t.m0 + rank * 128 + qd * 32 + lane + tap_shift(g, k.tap);
            if (px >= 0 && px < g.M) f = exp2_int(g.ea[px] - kRowShift);
          }
          const int kk = k16_of<T::ks>(g, k.c);
          for (int i0 = 0; i0 < kk; i0 += g.group, ++gi) {
            buf = gi % T::depth;
            if (!(ok = __all_sync(0xffffffffu, wait_or_abort(accfullb + buf * 8, (gi / T::depth) & 1, abortb)))) break;
            tc_fence_after_sync();
#pragma unroll
            for (int j0 = 0; j0 < NC; j0 += 16) {
              float v[16];
              tmem_ld16(taddr + buf * BN + j0, v);
              if (j0 + 16 == NC && (left > 1 || i0 + g.group < kk)) {
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) arrive_cluster(leader_addr(accfreeb + buf * 8));
              }
#pragma unroll
              for (int j = 0; j < 16; ++j) tot[j0 + j] = CONV ? fmaf(v[j], f, tot[j0 + j]) : tot[j0 + j] + v[j];
            }
          }
        }
      }
      if (!ok) break;
      // The totals go through the accumulator just read, so that a short loop stores them: unrolled over registers the
      // stores are 30 KB of code that every tile fetches anew: 8 us a tile (4096 x 4096 x 1024: 121 us, now 99).
#pragma unroll
      for (int j0 = 0; j0 < NC; j0 += 16) tmem_st16(taddr + buf * BN + j0, tot + j0);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      const UnitAt t = unit_at<BN, MN>(g, unit);   // again: cheaper than registers held through the loop
      const int row = rank * 128 + qd * 32 + lane, m = t.m0 + row;
      const bool cut = unit >= g.whole && g.splits > 1;
      long off = row;
      bool in = true;
      if (!cut) in = row_at<CONV>(g, m, &off);
      const long ldn = cut ? kBM : g.ldn;
      const int e = cut || MN ? 0 : CONV ? kRowShift : in ? g.ea[m] : 0, n0 = t.n0 + c0, N = cut ? t.n0 + BN : g.N;
      float* dst = cut ? g.partial + ((size_t)(unit - g.whole) * BN + c0) * kBM + off
                       : g.out + (size_t)t.tap * g.result + off + (long)n0 * ldn;
      const int* eb = g.eb + n0 + (lane & 15);
      int next = !MN && !cut && n0 + (lane & 15) < N ? *eb : 0;
#pragma unroll 1
      for (int j0 = 0; j0 < NC; j0 += 16) {
        float v[16];
        tmem_ld16(taddr + buf * BN + j0, v);
        const int ebv = next, left = N - n0 - j0;
        next = !MN && !cut && j0 + 16 + (lane & 15) < min(NC, N - n0) ? eb[j0 + 16] : 0;
        if (!MN) {
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = scale_by(v[j], e + __shfl_sync(0xffffffffu, ebv, j));
        }
        if (!CONV && g.vec && !cut) {   // 16-byte stores along a row
#pragma unroll
          for (int j = 0; j < 16; j += 4)
            if (in && j < left) *reinterpret_cast<float4*>(dst + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
          dst += 16;
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j, dst += ldn)
            if (in && j < left) *dst = v[j];
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) arrive_cluster(leader_addr(accfreeb + buf * 8));
      if constexpr (MN)
        if (*edges) edge_pixels<BN>(g, unit);
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (tid == 0 && *abort_flag) {
    atomicCAS(&g_gemm_tc_status, 0, (1 << 16) | (blockIdx.x & 0xffff));
    const long long t0 = clock64();   // copies in flight land before the shared memory is given back
    while (clock64() - t0 < 40000000ll) {
    }
  }
  cluster_sync();   // the peer's products read this CTA's shared memory, and its commits arrive on its barriers
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, T::tmem_cols);
  }
}

// The sums of a cut tile, in the order of K, and the exponents.  grid (cut tiles, BN / 8), one row per
// thread: enough CTAs to keep the L2 busy (34 tiles cut in two: 24 us with 32 columns per CTA, 6 with 8).
constexpr int kJoinCols = 8;
template <int BN, bool MN, bool CONV>
__global__ void __launch_bounds__(kBM) join_tiles_kernel(const __grid_constant__ SplitGemm g) {
  grid_dependency_wait();
  const UnitAt t = unit_at<BN, MN>(g, g.whole + blockIdx.x * g.splits);
  const int m = t.m0 + threadIdx.x;
  long off;
  if (!row_at<CONV>(g, m, &off)) return;
  const int e = MN ? 0 : CONV ? kRowShift : g.ea[m];
  const int n0 = t.n0 + blockIdx.y * kJoinCols;
  const float* src = g.partial + ((size_t)blockIdx.x * g.splits * BN + blockIdx.y * kJoinCols) * kBM + threadIdx.x;
  float* dst = g.out + (size_t)t.tap * g.result + off;
  float v[kJoinCols];
#pragma unroll
  for (int j = 0; j < kJoinCols; ++j) v[j] = __ldcs(src + j * kBM);
  for (int q = 1; q < g.splits; ++q)
#pragma unroll
    for (int j = 0; j < kJoinCols; ++j) v[j] += __ldcs(src + ((size_t)q * BN + j) * kBM);
#pragma unroll
  for (int j = 0; j < kJoinCols; ++j)
    if (n0 + j < g.N) dst[(long)(n0 + j) * g.ldn] = MN ? v[j] : scale_by(v[j], e + g.eb[n0 + j]);
}

// ---- operand planes -----------------------------------------------------------------------------------------------------
struct alignas(8) Half4 {
  __half2 a, b;
};
__device__ __forceinline__ void split4(float4 v, float sc, Half4& hi, Half4& lo) {
  v.x *= sc; v.y *= sc; v.z *= sc; v.w *= sc;
  hi.a = __floats2half2_rn(v.x, v.y);
  hi.b = __floats2half2_rn(v.z, v.w);
  const float2 p = __half22float2(hi.a), q = __half22float2(hi.b);
  lo.a = __floats2half2_rn(v.x - p.x, v.y - p.y);
  lo.b = __floats2half2_rn(v.z - q.x, v.w - q.y);
}
__device__ __forceinline__ unsigned max4(unsigned m, float4 v) {
  return max(max(max(m, abs_bits(v.x)), abs_bits(v.y)), max(abs_bits(v.z), abs_bits(v.w)));
}
// four values from c on of a row of `len`, zero past its end (`vec`: the row is 16-byte aligned).  Ordinary loads: the kernels here
// start while the one that writes the row may still run (the multiplied-out weight, or the result of another call), and the
// read-only path (__ldg) is for memory that nothing writes during the kernel's life.
__device__ __forceinline__ float4 load4(const float* row, int c, int len, bool vec) {
  if (vec && c + 4 <= len) return *reinterpret_cast<const float4*>(row + c);
  return make_float4(c < len ? row[c] : 0.f, c + 1 < len ? row[c + 1] : 0.f, c + 2 < len ? row[c + 2] : 0.f,
                     c + 3 < len ? row[c + 3] : 0.f);
}

// Both operands of a product are split in one launch: the CTAs below `first` take the first.
struct SplitJob {
  const float* src;
  int rows, segs, len, ld;   // rows of `segs` segments of `len` values, `ld` apart (columns and pixels: see the kernels)
  int ldo;                   // of a segment of the planes: a multiple of 8
  bool vec;
  uint16_t* hi;
  size_t plane;
  int* ex;
  int per;                   // rows of a CTA
};
struct SplitJobs {
  SplitJob job[2];
  int first;
};

// One exponent per row.  A warp takes a row of up to 512 values, a CTA a longer one; a row of up to 4096 values is read once.
__global__ void __launch_bounds__(256) split_rows_kernel(const __grid_constant__ SplitJobs jobs) {
  constexpr int Q = 4;
  __shared__ unsigned red[8];
  grid_dependency_wait();
  const bool second = (int)blockIdx.x >= jobs.first;
  const SplitJob& p = jobs.job[second];
  const int block = blockIdx.x - (second ? jobs.first : 0), segs = p.segs, len = p.len;
  const bool wide = segs * (long)len > 512;
  const int tpr = wide ? 256 : 32, sub = wide ? threadIdx.x : threadIdx.x & 31;
  const int row = wide ? block : block * 8 + (threadIdx.x >> 5);
  const bool in = row < p.rows;
  const int quads = (len + 3) / 4, n = in ? segs * quads : 0;
  const float* s = p.src + (size_t)row * segs * p.ld;
  float4 v[Q];
  unsigned mx = 0;
  auto at = [&](int i) {
    const int seg = segs == 1 ? 0 : i / quads;
    return load4(s + (size_t)seg * p.ld, (i - seg * quads) * 4, len, p.vec);
  };
  if (segs == 1 && p.vec && !(len & 3)) {   // no condition between the loads: 4096 x 4096 24.8 -> 22.4 us
#pragma unroll
    for (int q = 0; q < Q; ++q) v[q] = q * tpr + sub < n ? *reinterpret_cast<const float4*>(s + (q * tpr + sub) * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
  } else {
#pragma unroll
    for (int q = 0; q < Q; ++q) v[q] = q * tpr + sub < n ? at(q * tpr + sub) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
#pragma unroll
  for (int q = 0; q < Q; ++q) mx = max4(mx, v[q]);
  for (int i = Q * tpr + sub; i < n; i += tpr) mx = max4(mx, at(i));
  mx = __reduce_max_sync(0xffffffffu, mx);
  if (wide) {
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i) mx = max(mx, red[i]);
  }
  const int e = row_exponent(mx, kLeast);
  const float sc = exp2_int(-e);
  if (in && sub == 0) p.ex[row] = e;
  uint16_t* d = p.hi + (size_t)row * segs * p.ldo;
  auto put = [&](int i, float4 x) {
    const int seg = segs == 1 ? 0 : i / quads;
    const size_t o = (size_t)seg * p.ldo + (i - seg * quads) * 4;
    Half4 h, l;
    split4(x, sc, h, l);
    *reinterpret_cast<Half4*>(d + o) = h;
    *reinterpret_cast<Half4*>(d + p.plane + o) = l;
  };
#pragma unroll
  for (int q = 0; q < Q; ++q)
    if (q * tpr + sub < n) put(q * tpr + sub, v[q]);
  for (int i = Q * tpr + sub; i < n; i += tpr) put(i, at(i));
}

// [rows][len] as three bf16 planes.  Block (64, 4): 256 columns, every fourth row of a range.
__global__ void __launch_bounds__(256) split_columns_kernel(const __grid_constant__ SplitJobs jobs) {
  grid_dependency_wait();
  const bool second = (int)blockIdx.x >= jobs.first;
  const SplitJob& p = jobs.job[second];
  const int cols = p.len, c = (blockIdx.x - (second ? jobs.first : 0)) * 256 + threadIdx.x * 4;
  const int r0 = blockIdx.y * p.per, r1 = min(p.rows, r0 + p.per);
  if (c >= cols) return;
  const auto put = [&](int r, const float4& v) {
    const Bf3 x = split3(v.x, v.y), y = split3(v.z, v.w);
    uint16_t* d = p.hi + (size_t)r * p.ldo + c;
#pragma unroll
    for (int q = 0; q < 3; ++q) *reinterpret_cast<uint2*>(d + q * p.plane) = make_uint2(x.p[q], y.p[q]);
  };
  // Four rows of a thread in flight, without a condition between the loads: both operands of 4096 x 4096 52 -> 50 us.
  constexpr int B = 4;
  int r = r0 + threadIdx.y;
  if (p.vec && c + 4 <= cols)
    for (; r + 4 * (B - 1) < r1; r += 4 * B) {
      float4 v[B];
#pragma unroll
      for (int i = 0; i < B; ++i) v[i] = *reinterpret_cast<const float4*>(p.src + (size_t)(r + 4 * i) * cols + c);
#pragma unroll
      for (int i = 0; i < B; ++i) put(r + 4 * i, v[i]);
    }
#pragma unroll 4
  for (; r < r1; r += 4) put(r, load4(p.src + (size_t)r * cols, c, cols, p.vec));
}

// NCHW -> [n][pixel][channel] planes with padW zero pixels after each row and padH zero rows after each image: what a filter
// tap reads beside an image is then the end of the row or image before, and a tap is a shift of the row index, which TMA
// takes at any value (only the contiguous coordinate has an alignment rule).  Fp16 planes with an exponent per pixel, or
// (THREE) bf16 planes.  In a job: len = channels, rows = N (H + padH) (W + padW).
struct Images {
  int N, H, W, padH, padW;
  int* dropped;   // THREE: a word per 32 pixels of both operands (null: the filter has no ring)
};
// What bounds it is memory latency, so a thread has the loads of 32 channels of its pixel in flight and four CTAs share an SM; four channels of a
// pixel are together in shared memory (16-byte accesses, eight bytes of a plane per store).  32 images of 256 channels 28x28: pairs by pixel 14.9
// -> 11.6 us (with 16 loads in flight and channels apart; three or four CTAs alike, five 12.4).
constexpr int kPxTile = kGradKS, kPxPitch = kPxTile + 1;   // pitch: of four channels; a tile is a step of the gradient (see edge_pixels)
static_assert(kPxTile == 32, "");   // a pixel per lane
template <bool THREE>
__global__ void __launch_bounds__(256, 4) split_pixels_kernel(const __grid_constant__ SplitJobs jobs, const Images im) {
  extern __shared__ float px_smem[];
  __shared__ unsigned red[8][kPxTile];
  const bool second = (int)blockIdx.x >= jobs.first;
  const SplitJob& job = jobs.job[second];
  const int CH = job.len, HW = im.H * im.W;
  const int quads = (CH + 3) / 4;
  float4* tile = reinterpret_cast<float4*>(px_smem);      // [quads][kPxPitch]
  float* scale = px_smem + 4 * quads * kPxPitch;          // [kPxTile]
  const int Wp = im.W + im.padW, PP = (im.H + im.padH) * Wp, rows = job.rows;
  const int p0 = (blockIdx.x - (second ? jobs.first : 0)) * kPxTile, tx = threadIdx.x, ty = threadIdx.y, tid = ty * 32 + tx;
  grid_dependency_wait();
  {
    const int p = p0 + tx, n = p / PP, q = p - n * PP, h = q / Wp, w = q - h * Wp;
    const bool in = p < rows && h < im.H && w < im.W;
    const float* s = job.src + (((size_t)n * CH) * im.H + h) * im.W + w;
    unsigned m = 0;
    float most = 0.f;      // (three-way maxima of floats: a third of the instructions)
    constexpr int B = 8;   // quads of a thread whose loads are in flight together
    for (int k0 = ty; k0 < quads; k0 += 8 * B) {
      float v[B][4];
#pragma unroll
      for (int j = 0; j < B; ++j)
#pragma unroll
        for (int l = 0; l < 4; ++l) {
          const int c = (k0 + j * 8) * 4 + l;
          v[j][l] = in && c < CH ? s[(size_t)c * HW] : 0.f;
        }
#pragma unroll
      for (int j = 0; j < B; ++j)
        if (k0 + j * 8 < quads) {
          tile[(k0 + j * 8) * kPxPitch + tx] = make_float4(v[j][0], v[j][1], v[j][2], v[j][3]);
          if (THREE) most = most_nan(most_nan(most, v[j][0], v[j][1]), v[j][2], v[j][3]);
          else m = max(m, max(max(abs_bits(v[j][0]), abs_bits(v[j][1])), max(abs_bits(v[j][2]), abs_bits(v[j][3]))));
        }
    }
    if (THREE) {
      const bool edge = h < im.padH || h >= im.H - im.padH || w < im.padW || w >= im.W - im.padW, drop = im.dropped && edge && !(most <= FLT_MAX);
      if (drop)   // (see edge_pixels)
        for (int k = ty; k < quads; k += 8) {
          float4& v = tile[k * kPxPitch + tx];
          const auto finite = [](float f) { return abs_bits(f) < 0x7f800000u ? f : 0.f; };
          v = make_float4(finite(v.x), finite(v.y), finite(v.z), finite(v.w));
        }
      const int any = __syncthreads_or(drop);
      if (im.dropped && tid == 0) im.dropped[blockIdx.x] = any;
    } else {
      red[ty][tx] = m;
      __syncthreads();
    }
  }
  if (!THREE) {
    if (tid < kPxTile) {
      unsigned m = red[0][tid];
#pragma unroll
      for (int i = 1; i < 8; ++i) m = max(m, red[i][tid]);
      const int e = row_exponent(m, kLeastConv);
      scale[tid] = exp2_int(-e);
      if (p0 + tid < rows) job.ex[p0 + tid] = e;
    }
    __syncthreads();
  }
  const auto put = [&](int i, int k) {
    uint16_t* d = job.hi + (size_t)(p0 + i) * job.ldo + 4 * k;
    const float4 v = tile[k * kPxPitch + i];
    if (THREE) {
      const Bf3 x = split3(v.x, v.y), y = split3(v.z, v.w);
#pragma unroll
      for (int q = 0; q < 3; ++q) *reinterpret_cast<uint2*>(d + q * job.plane) = make_uint2(x.p[q], y.p[q]);
    } else {
      Half4 h, l;
      split4(v, scale[i], h, l);
      *reinterpret_cast<Half4*>(d) = h;
      *reinterpret_cast<Half4*>(d + job.plane) = l;
    }
  };
  if (quads > 16) {   // a warp writes the channels of a pixel, four per lane
    for (int k = tx; k < quads; k += 32) {
#pragma unroll
      for (int j = 0; j < kPxTile / 8; ++j) {
        const int i = ty + j * 8;
        if (p0 + i >= rows) break;
        put(i, k);
      }
    }
  } else {            // of several: pairs of 19 images of 32 channels 29x29 4.75 -> 4.27 us (4.19 where a lane had two channels)
    const int log = quads > 8 ? 4 : quads > 4 ? 3 : 2, k = tx & ((1 << log) - 1);
    for (int i = (ty * 32 + tx) >> log; i < kPxTile; i += 256 >> log)
      if (k < quads && p0 + i < rows) put(i, k);
  }
}

// ---- host ----------------------------------------------------------------------------------------------------------------
}  // namespace
// B200CP_GEMM_TC=0 keeps the CUDA-core products, 2 takes the tensor ones at every size (read per call: tests switch it)
int gemm_tc_mode() {
  const char* e = getenv("B200CP_GEMM_TC");
  return e && e[0] == '0' ? 0 : e && e[0] == '2' ? 2 : 1;
}
namespace {

// tensor of all planes: dimensions from the contiguous one outwards, strides in elements
int encode_planes(CUtensorMap* map, const uint16_t* base, int planes, const size_t (&dim)[3], const size_t (&stride)[2], size_t plane,
                  const unsigned (&box)[3]) {
  PFN_encodeTiled enc = get_encode_tiled();
  if (!enc) return fail(B200CP_ERR_NO_DEVICE, "cuTensorMapEncodeTiled entry point not available");
  const cuuint64_t gdim[4] = {dim[0], dim[1], dim[2], (cuuint64_t)planes};
  const cuuint64_t gstr[3] = {stride[0] * 2, stride[1] * 2, plane * 2};
  const cuuint32_t bx[4] = {box[0], box[1], box[2], (cuuint32_t)planes}, estr[4] = {1, 1, 1, 1};
  const CUresult cr = enc(map, planes == 3 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<uint16_t*>(base), gdim, gstr, bx, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (cr != CUDA_SUCCESS) return fail(B200CP_ERR_CUDA, "cuTensorMapEncodeTiled failed with code %d", (int)cr);
  return B200CP_OK;
}

// planes of one operand in the scratch: fp16 hi / lo with exponents, or three of bf16
struct Planes {
  uint16_t* hi;
  int* ex;
  size_t rows, plane;   // plane: values of one plane
  int ld;
};
size_t pair_floats(size_t rows, size_t ld, size_t exps) { return align_up(rows * ld, 64) + align_up(exps, 64); }
size_t dropped_words(size_t pixels) { return align_up(2 * ((pixels + kPxTile - 1) / kPxTile), 64); }
size_t triple_floats(size_t rows, size_t ld) { return align_up(rows * ld / 2 * 3, 64); }   // (ld is even)
Planes take_pair(float*& at, size_t rows, size_t ld, size_t exps) {
  Planes p{reinterpret_cast<uint16_t*>(at), nullptr, rows, rows * ld, (int)ld};
  p.ex = reinterpret_cast<int*>(at + align_up(rows * ld, 64));
  at += pair_floats(rows, ld, exps);
  return p;
}
Planes take_triple(float*& at, size_t rows, size_t ld) {
  const Planes p{reinterpret_cast<uint16_t*>(at), nullptr, rows, rows * ld, (int)ld};
  at += triple_floats(rows, ld);
  return p;
}
int ld8(int n) { return (n + 7) / 8 * 8; }

// (The kernels are programmatic dependents of one another; what comes before the first of a call is not this file's.)
SplitJob job_of(const float* src, int rows, int segs, int len, int ld, const Planes& p) {
  SplitJob j{};
  j.src = src; j.rows = rows; j.segs = segs; j.len = len; j.ld = ld;
  j.ldo = p.ld; j.hi = p.hi; j.plane = p.plane; j.ex = p.ex;
  j.vec = ld % 4 == 0 && !(reinterpret_cast<uintptr_t>(src) & 15);
  return j;
}
int split_rows(const SplitJob& a, const SplitJob& b, cudaStream_t st) {
  const auto ctas = [](const SplitJob& j) { return (long)j.segs * j.len > 512 ? j.rows : ceil_div(j.rows, 8); };
  SplitJobs jobs{{a, b}, ctas(a)};
  B200CP_CUDA_OK(launch_kernel(split_rows_kernel, dim3(ctas(a) + ctas(b)), dim3(256), 0, st, true, jobs));
  B200CP_LAUNCH_OK("split_rows_kernel");
  return B200CP_OK;
}
int split_columns(SplitJob a, SplitJob b, cudaStream_t st) {   // of the same number of rows
  a.per = b.per = std::max(16, ceil_div(a.rows, 64));
  SplitJobs jobs{{a, b}, ceil_div(a.len, 256)};
  B200CP_CUDA_OK(launch_kernel(split_columns_kernel, dim3(jobs.first + ceil_div(b.len, 256), ceil_div(a.rows, a.per)), dim3(64, 4), 0,
                               st, true, jobs));
  B200CP_LAUNCH_OK("split_columns_kernel");
  return B200CP_OK;
}
constexpr int kMostChannels = 1024;   // of split_pixels_kernel's tile: 139 KB
// the fp16 planes of one tensor, or (THREE) the bf16 planes of two
template <bool THREE>
int split_pixels(const SplitJob& a, const SplitJob& b, const Images& im, cudaStream_t st) {
  const SplitJobs jobs{{a, b}, ceil_div(a.rows, kPxTile)};
  const int most = std::max(a.len, b.len);
  const int channels = (most + 3) / 4 * 4;
  const size_t smem = sizeof(float) * ((size_t)channels * kPxPitch + kPxTile);
  static std::atomic<int> set[64];
  B200CP_CUDA_OK(ensure_dynamic_smem(reinterpret_cast<const void*>(split_pixels_kernel<THREE>), set, (int)smem));
  B200CP_CUDA_OK(launch_kernel(split_pixels_kernel<THREE>, dim3(jobs.first + ceil_div(b.rows, kPxTile)), dim3(32, 8), smem, st, true, jobs,
                               im));
  B200CP_LAUNCH_OK("split_pixels_kernel");
  return B200CP_OK;
}

// Accumulators of 64 terms, and of 32 where the sum has at most kShortSum steps.  Against float64 an accumulator of 32, 64, 128,
// 256 terms is cut off by about 0.5, 1.1, 4, 8e-7, and the roundings of n totals add 2.5e-8 sqrt(n / 2): 64 terms are best for
// long sums (2.2e-7 for 4096 terms; 32 terms: 2.5e-7, and the read-out falls behind the products), 32 for short ones.
constexpr int kShortSum = 16;
// Tiles of a product, and the cut of the tiles that do not fill the pairs (see SplitGemm).
struct TcTiles {
  int bn, tiles_m, tiles_n, whole, splits, steps, cut;   // cut: tiles that are cut
  double us;
};
// Measured us of a step (twelve instructions: 64 k, MN-major 32) and of a unit beside its steps.  128 and 64 columns are not in proportion: the rows of A are read
// from shared memory once per instruction, whatever its width.
double step_us(int bn) { return bn == 256 ? 1.35 : bn == 128 ? 0.95 : 0.7; }
constexpr double kUnitUs = 2.0;
TcTiles tc_tiles(long M, long N, int total, int results, bool mn, const DeviceInfo& di) {
  TcTiles best{};
  best.us = 1e300;
  const int pairs = di.sm_count / 2;
  for (int bn = 256; bn >= (mn ? 128 : 64); bn /= 2) {
    const long tm = (M + kBM - 1) / kBM, tn = (N + bn - 1) / bn, tiles = tm * tn * results;
    if (tiles > 0x3fffffff) continue;
    TcTiles t{bn, (int)tm, (int)tn, (int)(tiles / pairs * pairs), 1, total, (int)(tiles % pairs), 0.0};
    t.us = tiles / pairs * (total * step_us(bn) + kUnitUs);
    if (t.cut) {
      double tail = 1e300;
      for (int q = 1; q * t.cut <= pairs && (q == 1 || total / q >= 4); ++q) {
        const int steps = ceil_div(total, q);
        if ((q - 1) * steps >= total) continue;
        // a cut costs the launch that joins the sums, and their way through L2
        const double us = steps * step_us(bn) + kUnitUs + (q > 1 ? 3.0 + (double)t.cut * (q + 1) * kBM * bn * 4e-6 / 4.0 : 0.0);
        if (us < tail) { tail = us; t.splits = q; t.steps = steps; }
      }
      t.us += tail;
    }
    if (t.us < best.us) best = t;
  }
  return best;
}
size_t partial_floats(const TcTiles& t) { return t.splits > 1 ? (size_t)t.cut * t.splits * t.bn * kBM : 0; }

template <int BN, bool MN, bool CONV>
int launch_tile(const SplitGemm& g, int cut, const CUtensorMap& a, const CUtensorMap& b, const DeviceInfo& di, cudaStream_t st) {
  static std::atomic<int> set[64];
  B200CP_CUDA_OK(ensure_dynamic_smem(reinterpret_cast<const void*>(split_gemm_kernel<BN, MN, CONV>), set, (int)Tile<BN, MN>::smem));
  const int pairs = std::min(g.units, di.sm_count / 2);
  B200CP_CUDA_OK(launch_kernel(split_gemm_kernel<BN, MN, CONV>, dim3(2 * pairs), dim3(Tile<BN, MN>::threads),
                               Tile<BN, MN>::smem, st, true, g, a, b));
  B200CP_LAUNCH_OK("split_gemm_kernel");
  if (g.splits > 1) {
    B200CP_CUDA_OK(launch_kernel(join_tiles_kernel<BN, MN, CONV>, dim3(cut, BN / kJoinCols), dim3(kBM), 0, st, true, g));
    B200CP_LAUNCH_OK("join_tiles_kernel");
  }
  return B200CP_OK;
}
// g has the sizes, exponents and strides of the result; `partial` holds partial_floats(t)
int run_split_gemm(SplitGemm g, const TcTiles& t, size_t result, bool mn, bool conv, const CUtensorMap& a, const CUtensorMap& b,
                   float* out, float* partial, const DeviceInfo& di, cudaStream_t st) {
  g.tiles_m = t.tiles_m; g.tiles_n = t.tiles_n; g.whole = t.whole; g.splits = t.splits; g.steps = t.steps;
  g.units = t.whole + t.cut * t.splits;
  g.group = mn || g.total <= kShortSum ? 2 : 4;
  g.result = result;
  g.out = out;
  g.partial = partial;
#define TILE(BN, MN, CONV) launch_tile<BN, MN, CONV>(g, t.cut, a, b, di, st)
  if (mn) return t.bn == 256 ? TILE(256, true, false) : TILE(128, true, false);
  if (conv) return t.bn == 256 ? TILE(256, false, true) : t.bn == 128 ? TILE(128, false, true) : TILE(64, false, true);
  return t.bn == 256 ? TILE(256, false, false) : t.bn == 128 ? TILE(128, false, false) : TILE(64, false, false);
#undef TILE
}

}  // namespace

// ---- gradient products: both operands have the batch (or pixels) as rows -------------------------------------------------
// G[M][N] = A^T B with A [K][M], B [K][N]: rows of the kernel's result are the N columns of G, which are contiguous.
namespace {
TcTiles grad_tiles(int K, int M, int N, const DeviceInfo& di) { return tc_tiles(N, M, ceil_div(K, kGradKS), 1, true, di); }
// planes of an operand with K rows of n values
int encode_rows(CUtensorMap* map, const Planes& p, int n, size_t K) {
  return encode_planes(map, p.hi, 3, {(size_t)n, K, 1}, {(size_t)p.ld, p.plane}, p.plane, {64, kGradKS, 1});
}
}  // namespace

bool gemm_tc_supported(int K, int M, int N) {
  const int mode = gemm_tc_mode();
  return mode && (mode == 2 || (M >= 128 && N >= 128 && K >= 256)) && get_encode_tiled() != nullptr;
}

size_t gemm_tc_scratch_floats(int K, int M, int N) {
  DeviceInfo di;
  if (device_info(&di)) di.sm_count = 148;
  return triple_floats(K, ld8(M)) + triple_floats(K, ld8(N)) + partial_floats(grad_tiles(K, M, N, di));
}

int gemm_tc_launch(int K, int M, int N, const float* A, const float* B, float* G, float* scratch, cudaStream_t st) {
  DeviceInfo di;
  if (int rc = device_info(&di)) return rc;
  float* at = scratch;
  const Planes pn = take_triple(at, K, ld8(N)), pm = take_triple(at, K, ld8(M));
  if (int rc = split_columns(job_of(B, K, 1, N, N, pn), job_of(A, K, 1, M, M, pm), st)) return rc;
  CUtensorMap mn, mm;
  if (int rc = encode_rows(&mn, pn, N, K)) return rc;
  if (int rc = encode_rows(&mm, pm, M, K)) return rc;
  const TcTiles t = grad_tiles(K, M, N, di);
  SplitGemm g{};
  g.M = N; g.N = M; g.total = ceil_div(K, kGradKS); g.kc = g.total; g.Kc = K;
  g.FW = 1;
  g.ldm = 1; g.ldn = N;
  return run_split_gemm(g, t, (size_t)M * N, true, false, mn, mm, G, at, di, st);
}

// G[tap][t][c] = sum_{n,h,w} dV[n,t,h,w] * Xpad[n,c,h+y,w+x]: K = the pixels of the padded planes; the taps are as many
// products over the same planes, with the rows of X shifted.
namespace {
struct GradConv {
  int PP, taps;
  long K;
  TcTiles t;
};
bool grad_conv(GradConv& p, int N, int T, int C, int H, int W, int FH, int FW) {
  const int mode = gemm_tc_mode();
  if (!(mode && T <= kMostChannels && C <= kMostChannels && FH % 2 == 1 && FW % 2 == 1)) return false;
  p.PP = (H + (FH - 1) / 2) * (W + (FW - 1) / 2);
  p.taps = FH * FW;
  p.K = (long)N * p.PP;
  if (p.K > 0x3fffff00L || (mode == 1 && (p.K < 1024 || T < 128 || C < 128))) return false;
  DeviceInfo di;
  if (device_info(&di)) di.sm_count = 148;
  p.t = tc_tiles(C, T, (int)((p.K + kGradKS - 1) / kGradKS), p.taps, true, di);
  return get_encode_tiled() != nullptr;
}
}  // namespace

bool conv_gemm_tc_supported(int N, int T, int C, int H, int W, int FH, int FW) {
  GradConv p;
  return grad_conv(p, N, T, C, H, W, FH, FW);
}

size_t conv_gemm_tc_scratch_floats(int N, int T, int C, int H, int W, int FH, int FW) {
  GradConv p;
  if (!grad_conv(p, N, T, C, H, W, FH, FW)) return 0;
  return triple_floats(p.K, ld8(C)) + triple_floats(p.K, ld8(T)) + dropped_words(p.K) + partial_floats(p.t);
}

int conv_gemm_tc_launch(int N, int T, int C, int H, int W, int FH, int FW, const float* dV, const float* X, float* G,
                        float* scratch, cudaStream_t st) {
  GradConv p;
  if (!grad_conv(p, N, T, C, H, W, FH, FW)) return fail(B200CP_ERR_UNSUPPORTED, "tensor-core conv gradient: shape not taken");
  DeviceInfo di;
  if (int rc = device_info(&di)) return rc;
  const int padH = (FH - 1) / 2, padW = (FW - 1) / 2;
  float* at = scratch;
  const Planes px = take_triple(at, p.K, ld8(C)), pv = take_triple(at, p.K, ld8(T));
  int* dropped = padH || padW ? reinterpret_cast<int*>(at) : nullptr;
  at += dropped_words(p.K);
  if (int rc = split_pixels<true>(job_of(X, (int)p.K, 1, C, 0, px), job_of(dV, (int)p.K, 1, T, 0, pv), Images{N, H, W, padH, padW, dropped}, st))
    return rc;
  CUtensorMap mx, mv;
  if (int rc = encode_rows(&mx, px, C, p.K)) return rc;
  if (int rc = encode_rows(&mv, pv, T, p.K)) return rc;
  SplitGemm g{};
  g.M = C; g.N = T; g.total = ceil_div((int)p.K, kGradKS); g.kc = g.total; g.Kc = (int)p.K;
  g.FW = FW; g.padH = padH; g.padW = padW; g.Wp = W + padW;
  g.H = H; g.W = W; g.PP = p.PP;
  g.x = X; g.dv = dV; g.dropped = dropped;
  g.ldm = 1; g.ldn = C;
  return run_split_gemm(g, p.t, (size_t)T * C, true, false, mx, mv, G, at, di, st);
}

// ---- products with the multiplied-out weight --------------------------------------------------------------------------------
// Y[B][N] = X[B][K] W^T.  The rows of the kernel's result are the
// outputs (a warp then stores 32 neighbours of Y), or the batch where that leaves less of the tiles empty.
namespace {
struct DenseTc {
  TcTiles t;
  bool rows_are_batch;
};
DenseTc dense_tc(int B, int K, int N, const DeviceInfo& di) {
  const int total = ceil_div(K, kKS);
  const DenseTc a{tc_tiles(N, B, total, 1, false, di), false}, b{tc_tiles(B, N, total, 1, false, di), true};
  return b.t.us < 0.9 * a.t.us ? b : a;
}
// operand planes: a launch each, one pass that reads 4 bytes and writes 4
double split_us(double values) { return 2.5 + values * 8 / 4.5e6; }
}  // namespace

bool dense_tc_takes() { return gemm_tc_mode() && get_encode_tiled() != nullptr; }

double dense_tc_us(int B, int K, int N, const KronWeight& w) {
  DeviceInfo di;
  if (device_info(&di)) return 1e300;
  const double entries = (double)N * K;   // as planes, 2^24 entries: 38 us at R = 4, 42 at 32, 58 at 64, 213 at 256
  const double weight = kron_planes_takes(w.order, w.idims, w.odims, w.R, di.sm_count)
                            ? 8.0 + entries * (1.35e-6 + (w.R <= 64 ? 2.2e-8 : 4.0e-8) * w.R)
                            : kron_weight_us(w.order, w.idims, w.odims, w.R, 1, w.transposed) + split_us(entries);
  return 8.0 + weight + split_us((double)B * K) + dense_tc(B, K, N, di).t.us;
}

size_t dense_tc_scratch_floats(int B, int K, int N, const KronWeight& w) {
  DeviceInfo di;
  if (device_info(&di)) return 0;
  return (kron_planes_takes(w.order, w.idims, w.odims, w.R, di.sm_count) ? 0 : align_up((size_t)N * kron_weight_ld(K), 64)) +
         pair_floats(N, ld8(K), N) + pair_floats(B, ld8(K), B) + partial_floats(dense_tc(B, K, N, di).t);
}

int dense_tc_launch(int B, int K, int N, const float* X, const KronWeight& w, float* Y, float* scratch, cudaStream_t st) {
  DeviceInfo di;
  if (int rc = device_info(&di)) return rc;
  const DenseTc d = dense_tc(B, K, N, di);
  const bool direct = kron_planes_takes(w.order, w.idims, w.odims, w.R, di.sm_count);
  float *at = scratch, *W = scratch;
  if (!direct) at += align_up((size_t)N * kron_weight_ld(K), 64);
  const Planes pw = take_pair(at, N, ld8(K), N), px = take_pair(at, B, ld8(K), B);
  if (direct) {
    if (int rc = kron_planes_launch(w.order, w.idims, w.odims, w.R, w.F, w.transposed, pw.ld, pw.hi, pw.plane, pw.ex, st)) return rc;
    if (int rc = split_rows(job_of(X, B, 1, K, K, px), SplitJob{}, st)) return rc;
  } else {
    if (int rc = kron_weight_launch(w.order, w.idims, w.odims, w.R, w.F, nullptr, 1, w.transposed, false, W, st)) return rc;
    if (int rc = split_rows(job_of(W, N, 1, K, kron_weight_ld(K), pw), job_of(X, B, 1, K, K, px), st)) return rc;
  }
  const Planes &pa = d.rows_are_batch ? px : pw, &pb = d.rows_are_batch ? pw : px;
  CUtensorMap ma, mb;
  if (int rc = encode_planes(&ma, pa.hi, 2, {(size_t)K, 1, pa.rows}, {(size_t)pa.ld, (size_t)pa.ld}, pa.plane, {64, 1, 128})) return rc;
  if (int rc = encode_planes(&mb, pb.hi, 2, {(size_t)K, 1, pb.rows}, {(size_t)pb.ld, (size_t)pb.ld}, pb.plane,
                             {64, 1, (unsigned)d.t.bn / 2})) return rc;
  SplitGemm g{};
  g.M = (int)pa.rows; g.N = (int)pb.rows; g.total = ceil_div(K, kKS); g.kc = g.total; g.Kc = K;
  g.FW = 1;
  g.ea = pa.ex; g.eb = pb.ex;
  g.ldm = d.rows_are_batch ? N : 1;
  g.ldn = d.rows_are_batch ? 1 : N;
  g.vec = d.rows_are_batch && N % 4 == 0 && !(reinterpret_cast<uintptr_t>(Y) & 15);
  return run_split_gemm(g, d.t, 0, false, false, ma, mb, Y, at, di, st);
}

// V[n,t,h,w] = sum_{c,y,x} W[t][y,x][c] X[n,c,h+y-1,w+x-1] (3 x 3): rows are the padded pixels, and a
// step is 64 channels of one tap.
namespace {
constexpr int kPad = 1, kTaps = 9;
TcTiles conv_tc(int N, int C, int T, int H, int W, const DeviceInfo& di) {
  return tc_tiles((long)N * (H + kPad) * (W + kPad), T, kTaps * ceil_div(C, kKS), 1, false, di);
}
}  // namespace

bool conv_tc_takes(int N, int C, int T, int H, int W) {
  return gemm_tc_mode() && C <= kMostChannels && (long)N * (H + kPad) * (W + kPad) < 0x3fffff00L && get_encode_tiled() != nullptr;
}

double conv_tc_us(int N, int C, int T, int H, int W) {
  DeviceInfo di;
  if (device_info(&di)) return 1e300;
  return 8.0 + split_us((double)T * C * kTaps) + split_us((double)N * (H + kPad) * (W + kPad) * C) + conv_tc(N, C, T, H, W, di).us;
}

size_t conv_tc_scratch_floats(int N, int C, int T, int H, int W) {
  DeviceInfo di;
  if (device_info(&di)) return 0;
  const size_t px = (size_t)N * (H + kPad) * (W + kPad);
  return align_up((size_t)T * kTaps * kron_weight_ld(C), 64) + pair_floats(T, (size_t)kTaps * ld8(C), T) + pair_floats(px, ld8(C), px) +
         partial_floats(conv_tc(N, C, T, H, W, di));
}

int conv_tc_launch(int N, int C, int T, int H, int W, const float* X, const KronWeight& w, float* V, float* scratch,
                   cudaStream_t st) {
  DeviceInfo di;
  if (int rc = device_info(&di)) return rc;
  const TcTiles t = conv_tc(N, C, T, H, W, di);
  const int Wp = W + kPad, PP = (H + kPad) * Wp;
  const size_t px = (size_t)N * PP, ldk = ld8(C);
  const int ldw = kron_weight_ld(C);
  float *Wt = scratch, *at = scratch + align_up((size_t)T * kTaps * ldw, 64);
  if (int rc = kron_weight_launch(w.order, w.idims, w.odims, w.R, w.F, w.S, kTaps, w.transposed, w.flip, Wt, st)) return rc;
  Planes pw = take_pair(at, T, kTaps * ldk, T), pa = take_pair(at, px, ldk, px);
  pw.ld = (int)ldk;
  const SplitJob none{};
  if (int rc = split_rows(job_of(Wt, T, kTaps, C, ldw, pw), none, st)) return rc;
  if (int rc = split_pixels<false>(job_of(X, (int)px, 1, C, 0, pa), none, Images{N, H, W, kPad, kPad, nullptr}, st)) return rc;
  CUtensorMap ma, mb;
  if (int rc = encode_planes(&ma, pa.hi, 2, {(size_t)C, 1, px}, {ldk, ldk}, pa.plane, {64, 1, 128})) return rc;
  if (int rc = encode_planes(&mb, pw.hi, 2, {(size_t)C, kTaps, (size_t)T}, {ldk, kTaps * ldk}, pw.plane, {64, 1, (unsigned)t.bn / 2}))
    return rc;
  SplitGemm g{};
  g.M = (int)px; g.N = T; g.kc = ceil_div(C, kKS); g.total = kTaps * g.kc; g.Kc = C;
  g.FW = 3; g.padH = g.padW = kPad; g.Wp = Wp;
  g.ea = pa.ex; g.eb = pw.ex;
  g.ldn = (long)H * W;
  g.H = H; g.W = W; g.PP = PP;
  return run_split_gemm(g, t, 0, false, true, ma, mb, V, at, di, st);
}

// Reads (and clears) the status word of the GEMM kernel; the caller has synchronised the device.
int gemm_tc_status(int* out) {
  int v = 0, zero = 0;
  B200CP_CUDA_OK(cudaMemcpyFromSymbol(&v, g_gemm_tc_status, sizeof(int)));
  if (v) B200CP_CUDA_OK(cudaMemcpyToSymbol(g_gemm_tc_status, &zero, sizeof(int)));
  *out = v;
  return B200CP_OK;
}

}  // namespace b200cp
