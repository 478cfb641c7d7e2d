// Factor gradients from a large dense gradient G on the tensor cores: the modes (contract_peel.cu) in two halves of at most two modes
// each, a and b, whose vectors multiplied out are VA[a][r] and VB[b][r].  One pass over G gives both
//   SA[a][r] = sum_b G[a][b] VB[b][r],   SB[b][r] = sum_a G[a][b] VA[a][r],
// tensors smaller than G by the size of a half, from which the gradient of each mode is a sum over the other mode of its half.
// Peeled mode by mode, G costs the same 2 |G| R multiply-adds on FFMA, a tensor of |G| / |last mode| entries of R ranks is written and
// read again, and the products of the outer vectors are formed for every row of G.
//
// A CTA has 128 entries of a and walks tiles of 64 entries of b.  A tile of G is split into three bf16 parts (tc_common.cuh) once; it is the
// K-major A operand of the first product and the MN-major B operand of the second, whose A operand are the parts of VA:
//   D1[128 a][4 x 32] = G_hi (V_hi | V_mid | V_low | 0) + G_mid (0 | V_hi | V_mid | V_low) + G_low (0 | 0 | V_hi | V_mid)    K = 64
//   D2[part, r][64 b | 64 b]  = V_part (G_hi | G_mid + G_low)                                                            K = 128
// so the parts of V share an instruction, G_hi and G_mid one of twice the columns in D2.  D1 is added to totals in registers after each
// tile, D2 goes out as a partial sum per 128 entries of a: no accumulator is longer than 64 (D1) or 128 terms.  First parts of six bits (split3_short), so
// that the tensor core cuts next to nothing off, and the smaller parts have sums of their own.  Error of a factor's gradient against float64 over that of the
// peeled sums, 40 drawn layers: normally distributed values 0.69 (at most 0.95), positive ones 0.95 (1.15); with first parts of eight bits 0.88 (1.43) and
// 1.52 (2.97), the pass 1 % faster.
// G and the vectors are lifted by 2^17 (as in kron_small.cu: the third part of a value is 2^-16 of it).  A tile in which one of them is above 2^43 or
// infinite, or a product of two vectors below the smallest normal number, is multiplied in fp32 instead, one vector after the other (exact_tile).  (A NaN
// makes the same sums NaN either way.)
//
// What bounds it: the phases of a tile follow one another, load - split - products - sums, and two CTAs per SM overlap only in part (issue 45 %,
// shared memory 47 %, tensor pipe 22 %, DRAM 16 %; a tile takes 5000 cycles of an SM, of which G's 32 KB need 1400 and the
// products, bound by what they read from shared memory, 1700).  G of 4096 x 4096 at R = 32: 52 us and 12 for the sums, mode by mode 104 + 26 + 9;
// the layer's step with a batch of 4096 1812 -> 1699 us with the weight's planes of kron_small.cu.  5x13x11 -> 13x7x7 at R = 246 362 -> 130 us.
#include <algorithm>
#include <cfloat>

#include "contract.cuh"
#include "tc_common.cuh"

namespace b200cp {

namespace {

__device__ int g_halves_status = 0;   // 0 ok; otherwise (1 << 16) | (block index & 0xffff): a bounded wait ran out

constexpr int kHT = 256, kHA = 128, kHB = 64, kHR = 32;   // threads; entries of a and b and ranks of a tile
constexpr int kPlaneG = kHA * 128, kVBlock = 3 * kHR * 128;   // bytes of a part of G, of the parts of V for 64 entries
constexpr float kDrop = 1.f / (tc::kLift * tc::kLift), kLeastProduct = FLT_MIN * tc::kLift, kMost = 1.152921504606846976e18f;   // 2^60: no sum of 128 products overflows
constexpr size_t kHalvesSmem = 1024 + 3 * kPlaneG + 3 * kVBlock + kHR * 128;
// The second product reads 128 rows of the 96 that VA's blocks have: the others are the block behind, VB's after the last, and
// their results stay unread.
static_assert(kVBlock % 1024 == 0 && 128 * 128 <= 2 * kVBlock, "");

struct Half {
  int n, size;
  PeelMode m[2];
};
struct HalvesGeom {
  Half a, b;
  int R, btiles, splits; // tiles of b, and the CTAs that share them
  const float* G;
  float *sa, *sb;        // [splits][a.size][R], [tiles of a][b.size][R]
};

// Entry i of a half, the t digits slow and the c digits fast, so that consecutive ones are neighbours in G: its offset in G and its entry
// of each mode.
__device__ __forceinline__ int half_entry(const Half& h, int i, int (&e)[2]) {
  int off = 0;
  e[0] = e[1] = 0;
#pragma unroll
  for (int k = 1; k >= 0; --k)
    if (k < h.n) {
      const int q = i / h.m[k].nc, c = i - q * h.m[k].nc;
      i = q;
      off += c * (int)h.m[k].gc;
      e[k] = c * h.m[k].nt;
    }
#pragma unroll
  for (int k = 1; k >= 0; --k)
    if (k < h.n) {
      const int q = i / h.m[k].nt, t = i - q * h.m[k].nt;
      i = q;
      off += t * (int)h.m[k].gt;
      e[k] += t;
    }
  return off;
}
struct HalfTable {   // of a tile
  int off[kHA], e[kHA][2];
};

// A tile in fp32, the inner mode first as in contract_peel.cu: SB's sums to `out`, SA's to shared memory [r][a].  `sm` has the room of G's parts (G by
// [a][b], then the values of b's outer mode by [b][r]), `inner` that of the parts of VB.  G of 4096 x 4096 at R = 32, all tiles this way: 430 us instead of 54.
constexpr int kExactPitch = kHB + 4;
static_assert((kHA * kExactPitch + kHB * kHR) * 4 <= 3 * kPlaneG && kHB * kHR * 4 <= kVBlock, "");
__device__ __noinline__ void exact_tile(const HalvesGeom& g, float* sm, float* inner, const HalfTable& ta, const int* offb, const int (*eb)[2], int r0,
                                        float* out) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, r = r0 + lane, rv = min(r, g.R - 1);
  float *G = sm, *v0 = sm + kHA * kExactPitch, *v1 = inner;
  const float *b0 = g.b.m[0].vec + rv, *b1 = g.b.m[g.b.n - 1].vec + rv, *a0 = g.a.m[0].vec + rv, *a1 = g.a.m[g.a.n - 1].vec + rv;
#pragma unroll 8
  for (int i = tid; i < kHA * kHB; i += kHT) {
    const int a = i / kHB, b = i % kHB, oa = ta.off[a], ob = offb[b];
    G[a * kExactPitch + b] = oa >= 0 && ob >= 0 ? g.G[oa + ob] : 0.f;
  }
#pragma unroll
  for (int b = warp; b < kHB; b += 8) {   // (past the end G is 0, and so are they: 0 times infinity)
    v0[b * kHR + lane] = offb[b] >= 0 ? b0[(size_t)eb[b][0] * g.R] : 0.f;
    v1[b * kHR + lane] = g.b.n > 1 && offb[b] >= 0 ? b1[(size_t)eb[b][1] * g.R] : 1.f;
  }
  __syncthreads();
  float v[8];   // of entries 8 * warp on of b
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = 0.f;
  for (int a8 = 0; a8 < kHA; a8 += 8) {
    float x[8], y[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int a = a8 + q;
      x[q] = ta.off[a] >= 0 ? a0[(size_t)ta.e[a][0] * g.R] : 0.f;
      y[q] = ta.off[a] >= 0 && g.a.n > 1 ? a1[(size_t)ta.e[a][1] * g.R] : 1.f;
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const float4 *p = reinterpret_cast<const float4*>(G + (a8 + q) * kExactPitch + 8 * warp), c = p[0], d = p[1];
      const float w[8] = {c.x, c.y, c.z, c.w, d.x, d.y, d.z, d.w};
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = fmaf(w[i] * y[q], x[q], v[i]);
    }
  }
  if (r < g.R)
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (offb[8 * warp + i] >= 0) out[(size_t)(8 * warp + i) * g.R + lane] = v[i];
  const int a = (warp & 3) * 32 + lane, j0 = (warp >> 2) * 16;
  float w[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) w[j] = 0.f;
  for (int b4 = 0; b4 < kHB; b4 += 4) {
    const float4 c = *reinterpret_cast<const float4*>(G + a * kExactPitch + b4);
    const float x[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
      for (int j = 0; j < 16; j += 4) {
        const float4 y = *reinterpret_cast<const float4*>(v1 + (b4 + b) * kHR + j0 + j), z = *reinterpret_cast<const float4*>(v0 + (b4 + b) * kHR + j0 + j);
        w[j] = fmaf(x[b] * y.x, z.x, w[j]);
        w[j + 1] = fmaf(x[b] * y.y, z.y, w[j + 1]);
        w[j + 2] = fmaf(x[b] * y.z, z.z, w[j + 2]);
        w[j + 3] = fmaf(x[b] * y.w, z.w, w[j + 3]);
      }
  }
  __syncthreads();   // G and the values are read
#pragma unroll
  for (int j = 0; j < 16; ++j) sm[(j0 + j) * kHA + a] = w[j];
  __syncthreads();
}

// VEC: rows of four entries of b are neighbours in G and 16-byte aligned
template <bool VEC>
__global__ void __launch_bounds__(kHT, 2) halves_kernel(const __grid_constant__ HalvesGeom g) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t *va = sm + 3 * kPlaneG, *vb = va + 2 * kVBlock;
  __shared__ HalfTable ta;
  __shared__ int tboff[3][kHB], tbe[3][kHB][2];   // of this tile of b, the next and the one after
  __shared__ __align__(8) uint64_t done;
  __shared__ uint32_t tmem_slot;
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), quarter = warp & 3, grp = warp >> 2;
  const int a0 = blockIdx.x * kHA, t0 = (int)((long)blockIdx.y * g.btiles / g.splits), steps = (int)((long)(blockIdx.y + 1) * g.btiles / g.splits) - t0, r0 = blockIdx.z * kHR, r = r0 + lane;
  const int arows = min(kHA, g.a.size - a0);
  if (tid == 0) {
    tc::mbar_init(&done, 1);
    tc::fence_barrier_init();
  }
  if (warp == 0) tc::tmem_alloc(&tmem_slot, 256);
  auto table_b = [&](int s, int i) {   // entry i of tile s
    const int b = (t0 + s) * kHB + i;
    int e[2];
    const int off = b < g.b.size ? half_entry(g.b, b, e) : -1;
    tboff[s % 3][i] = off;
    tbe[s % 3][i][0] = off < 0 ? 0 : e[0];
    tbe[s % 3][i][1] = off < 0 ? 0 : e[1];
  };
  if (tid < kHA) {
    int e[2] = {0, 0};
    ta.off[tid] = tid < arows ? half_entry(g.a, a0 + tid, e) : -1;
    ta.e[tid][0] = e[0];
    ta.e[tid][1] = e[1];
  } else if (tid < kHA + kHB) {
    table_b(0, tid - kHA);
  } else {
    table_b(1, tid - kHA - kHB);
  }
  tc::tc_fence_before_sync();
  __syncthreads();
  tc::tc_fence_after_sync();
  const uint32_t tmem = tmem_slot, lanes = tmem + ((uint32_t)(quarter * 32) << 16);
  // 64 entries of a half as parts, [part, r][entry]: a warp has eight entries, a lane a rank and two of them at a time, which its
  // eighth of the warp (rows of the same banks) begins with
  const auto entry = [&](int i) { return 8 * warp + 2 * ((i + (lane >> 3)) & 3); };
  // (no load depends on a condition: with conditions they follow one another, 4000 cycles a tile)
  float y[4][2], f[4][2];
  const int rv = min(r, g.R - 1);
  auto load_values = [&](const Half& h, const int (*e)[2]) {
    const float *v0 = h.m[0].vec + rv, *v1 = (h.n > 1 ? h.m[1].vec : h.m[0].vec) + rv;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int k = entry(i) + j;
        y[i][j] = v0[e[k][0] * g.R];
        f[i][j] = v1[e[k][1] * g.R];
      }
  };
  auto multiply_values = [&](const Half& h, const int* off) {   // true: a value is out of the range of the parts
    float p[4][2], most = 0.f, least = FLT_MAX;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        p[i][j] = y[i][j] * tc::kLift;
        if (h.n > 1) p[i][j] *= f[i][j];
      }
      most = tc::most_of(most, p[i][0], p[i][1]);
      least = tc::least_of(least, p[i][0], p[i][1]);
    }
    bool out = most >= kMost;
    if (h.n > 1 && least < kLeastProduct)
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) out = out || (fabsf(p[i][j]) < kLeastProduct && y[i][j] != 0.f && f[i][j] != 0.f);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) y[i][j] = r < g.R && off[entry(i) + j] >= 0 ? p[i][j] : 0.f;
    return out;
  };
  auto split_values = [&](uint8_t* block) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int k = entry(i);
      const tc::Bf3 w = tc::split3_short<false>(y[i][0], y[i][1]);
      uint8_t* d = block + lane * 128 + ((((k >> 3) ^ lane) & 7) << 4) + (k & 7) * 2;
#pragma unroll
      for (int p = 0; p < 3; ++p) *reinterpret_cast<uint32_t*>(d + p * kHR * 128) = w.p[p];
    }
  };
  reinterpret_cast<uint4*>(vb + kVBlock)[tid] = make_uint4(0, 0, 0, 0);   // (32 rows)
  load_values(g.a, ta.e);
  bool outa = multiply_values(g.a, ta.off);
  split_values(va);
  load_values(g.a, ta.e + 64);
  outa = multiply_values(g.a, ta.off + 64) || outa;
  split_values(va + kVBlock);

  const uint64_t d0 = tc::make_smem_desc(0, 16, 1024, tc::kSwizzle128B);
  constexpr uint32_t idesc2 = tc::make_idesc_bf16(2 * kHB) | (1u << 16), idesc3 = tc::make_idesc_bf16(kHB) | (1u << 16);   // the B operand MN-major
  float tot[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) tot[j] = 0.f;
  bool fine = true;
  // A warp has two times eight entries of a; those of the next tile are on their way during the products of this one.
  float x[2][16];
  auto load_tile = [&](int s) {
    const int* off = tboff[s % 3];
    const int ob0 = off[VEC ? (lane & 15) * 4 : lane * 2], ob1 = VEC ? 0 : off[lane * 2 + 1];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int* oa = ta.off + (warp + 8 * i) * 8 + (VEC ? lane >> 4 : 0);
      if constexpr (VEC) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float4 v = oa[2 * k] >= 0 && ob0 >= 0 ? *reinterpret_cast<const float4*>(g.G + oa[2 * k] + ob0) : make_float4(0.f, 0.f, 0.f, 0.f);
          x[i][4 * k] = v.x; x[i][4 * k + 1] = v.y; x[i][4 * k + 2] = v.z; x[i][4 * k + 3] = v.w;
        }
      } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          x[i][2 * k] = oa[k] >= 0 && ob0 >= 0 ? g.G[oa[k] + ob0] : 0.f;
          x[i][2 * k + 1] = oa[k] >= 0 && ob1 >= 0 ? g.G[oa[k] + ob1] : 0.f;
        }
      }
    }
  };
  load_values(g.b, tbe[0]);
  bool outb = multiply_values(g.b, tboff[0]);
  grid_dependency_wait();   // G
  load_tile(0);
  for (int s = 0, issued = 0; s < steps; ++s) {
    float most = 0.f;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 16; j += 2) {
        x[i][j] *= tc::kLift;
        x[i][j + 1] *= tc::kLift;
        most = tc::most_of(most, x[i][j], x[i][j + 1]);
      }
    const bool out = outa || outb || most >= kMost;
    split_values(vb);
    load_values(g.b, tbe[(s + 1) % 3]);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float* v = x[i];
      uint8_t* d = sm + (warp + 8 * i) * 8 * 128;
      if constexpr (VEC) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const tc::Bf3 w0 = tc::split3_short<false>(v[4 * k], v[4 * k + 1]),
                        w1 = tc::split3_short<false>(v[4 * k + 2], v[4 * k + 3]);
          const int row = 2 * k + (lane >> 4);
          uint8_t* o = d + row * 128 + ((((lane & 15) >> 1) ^ row) << 4) + (lane & 1) * 8;
#pragma unroll
          for (int p = 0; p < 3; ++p) *reinterpret_cast<uint2*>(o + p * kPlaneG) = make_uint2(w0.p[p], w1.p[p]);
        }
      } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const tc::Bf3 w = tc::split3_short<false>(v[2 * k], v[2 * k + 1]);
          uint8_t* o = d + k * 128 + (((lane >> 2) ^ k) << 4) + (lane & 3) * 4;
#pragma unroll
          for (int p = 0; p < 3; ++p) *reinterpret_cast<uint32_t*>(o + p * kPlaneG) = w.p[p];
        }
      }
    }
    tc::fence_proxy_async();
    const bool exact = __syncthreads_or(out);
    if (!exact && warp == 0 && tc::elect_one()) {
      tc::tc_fence_after_sync();
      const uint64_t gd2 = tc::make_smem_desc(0, kPlaneG, 1024, tc::kSwizzle128B) + (tc::smem_u32(sm) >> 4);   // (64 rows on: the next part)
      const uint64_t gd = d0 + (tc::smem_u32(sm) >> 4), ad = d0 + (tc::smem_u32(va) >> 4), bd = d0 + (tc::smem_u32(vb) >> 4);
#pragma unroll
      for (int k = 0; k < kHB / 16; ++k) {
        tc::mma_f16_ss(tmem, gd + k * 2, bd + k * 2, tc::make_idesc_bf16(4 * kHR), k > 0);
        tc::mma_f16_ss(tmem + kHR, gd + (kPlaneG >> 4) + k * 2, bd + k * 2, tc::make_idesc_bf16(3 * kHR), true);
        tc::mma_f16_ss(tmem + 2 * kHR, gd + 2 * (kPlaneG >> 4) + k * 2, bd + k * 2, tc::make_idesc_bf16(2 * kHR), true);
      }
#pragma unroll
      for (int k = 0; k < kHA / 16; ++k) {   // 16 entries of a: 2048 bytes of G's rows, 32 of VA's
        const uint64_t av = ad + (k >> 2) * (kVBlock >> 4) + (k & 3) * 2;
        tc::mma_f16_ss(tmem + 4 * kHR, av, gd2 + k * 128, idesc2, k > 0);
        tc::mma_f16_ss(tmem + 4 * kHR + kHB, av, gd2 + 2 * (kPlaneG >> 4) + k * 128, idesc3, true);
      }
      tc::mma_commit(&done);
    }
    __syncwarp();
    if (s + 1 < steps) load_tile(s + 1);
    outb = multiply_values(g.b, tboff[(s + 1) % 3]);
    if (tid >= kHT - kHB) table_b(s + 2, tid - (kHT - kHB));
    float* dst = g.sb + ((size_t)blockIdx.x * g.b.size + (size_t)(t0 + s) * kHB) * g.R + r0;
    float* sums = reinterpret_cast<float*>(sm);
    if (exact) {
      exact_tile(g, sums, reinterpret_cast<float*>(vb), ta, tboff[s % 3], tbe[s % 3], r0, dst);
#pragma unroll
      for (int j = 0; j < 16; ++j) tot[j] += sums[(grp * 16 + j) * kHA + quarter * 32 + lane];
      __syncthreads();   // the sums are read
      continue;
    }
    fine = tc::mbar_wait(&done, issued++ & 1) && fine;   // (the other CTA of the SM works meanwhile)
    __syncwarp();
    tc::tc_fence_after_sync();
    {   // sums by [part][b][r]: the parts of G are used up
      float v[16], w[16];
      tc::tmem_ld16(lanes + 3 * kHR + grp * 16, v);
      tc::tmem_ld16(lanes + 2 * kHR + grp * 16, w);
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] += w[j];
      tc::tmem_ld16(lanes + kHR + grp * 16, w);
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] += w[j];
      tc::tmem_ld16(lanes + grp * 16, w);
#pragma unroll
      for (int j = 0; j < 16; ++j) tot[j] = fmaf(w[j] + v[j], kDrop, tot[j]);
      if (quarter < 3) {
#pragma unroll
        for (int j0 = 0; j0 < 32; j0 += 16) {
          tc::tmem_ld16(lanes + 4 * kHR + grp * 32 + j0, v);
          tc::tmem_ld16(lanes + 4 * kHR + kHB + grp * 32 + j0, w);
#pragma unroll
          for (int j = 0; j < 16; ++j) sums[(quarter * kHB + grp * 32 + j0 + j) * kHR + lane] = v[j] + w[j];
        }
      }
    }
    tc::tc_fence_before_sync();
    __syncthreads();   // and the accumulators are free
    const int* off = tboff[s % 3];
    if (r < g.R) {
#pragma unroll
      for (int i = 0; i < kHB / 8; ++i) {
        const float* p = sums + (warp + i * 8) * kHR + lane;
        if (off[warp + i * 8] >= 0) dst[(size_t)(warp + i * 8) * g.R + lane] = (p[0] + (p[kHB * kHR] + p[2 * kHB * kHR])) * kDrop;
      }
    }
    __syncthreads();   // the sums are read
  }
  if (!fine) atomicCAS(&g_halves_status, 0, (1 << 16) | (blockIdx.x & 0xffff));
  grid_launch_dependents();
  const int a = quarter * 32 + lane;
  if (a < arows) {
    float* out = g.sa + ((size_t)blockIdx.y * g.a.size + a0 + a) * g.R + r0 + grp * 16;
    const int have = g.R - r0 - grp * 16;
#pragma unroll
    for (int j = 0; j < 16; ++j)
      if (j < have) out[j] = tot[j];
  }
  tc::tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc::tc_fence_after_sync();
    tc::tmem_dealloc(tmem, 256);
  }
}

// ---- the halves' tensors and from them the gradients ----------------------------------------------------------------------------
struct HalvesSums {
  Half h[2];
  const float* part[2];
  float* dst[2];         // by the factor's own entries, [e0][e1][R]; of a half of one mode its gradient
  float* grad[2][2];
  int parts[2], R, blocks0;   // blocks of the first half's sums
};
constexpr int kManyParts = 64;

// The partial sums of an entry of a half: a warp, or where there are many eight, of which each has every eighth.
__global__ void __launch_bounds__(256) halves_sum_kernel(const __grid_constant__ HalvesSums g) {
  __shared__ float red[8][32];
  const int k = blockIdx.x >= g.blocks0, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, many = g.parts[k] > kManyParts;
  const int block = k ? blockIdx.x - g.blocks0 : blockIdx.x, i = many ? block : block * 8 + warp, r = blockIdx.y * 32 + lane;
  const Half& h = g.h[k];
  int e[2];
  half_entry(h, i, e);
  const size_t row = h.n > 1 ? (size_t)e[0] * (h.m[1].nc * h.m[1].nt) + e[1] : e[0], stride = (size_t)h.size * g.R;
  const bool in = i < h.size && r < g.R;
  grid_dependency_wait();
  const float* src = g.part[k] + (size_t)i * g.R + r;
  // eight at a time, their sum first: one after the other 64 parts would be off by 7e-8
  const int step = many ? 8 : 1, p0 = many ? warp : 0;
  const size_t next = step * stride;
  const float* q = src + p0 * stride;
  float v = 0.f;
  if (in) {
    int left = (g.parts[k] - p0 + step - 1) / step;
    for (; left >= 8; left -= 8, q += 8 * next) {
      float s[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) s[j] = q[j * next];
#pragma unroll
      for (int w = 4; w; w >>= 1)
#pragma unroll
        for (int j = 0; j < w; ++j) s[j] += s[j + w];
      v += s[0];
    }
    float rest = 0.f;
#pragma unroll 4
    for (; left > 0; --left, q += next) rest += *q;
    v += rest;
  }
  if (many) {
    red[warp][lane] = v;
    __syncthreads();
    if (warp) return;
#pragma unroll
    for (int w = 1; w < 8; ++w) v += red[w][lane];
  }
  if (in) g.dst[k][row * g.R + r] = v;
}

// a mode's entry of 32 ranks per CTA: the sum over the other mode of its half
__global__ void __launch_bounds__(256) halves_factor_kernel(const __grid_constant__ HalvesSums g) {
  __shared__ float red[8][32];
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5, r = blockIdx.y * 32 + x;
  int i = blockIdx.x, k = 0, m = 0;
  for (; k < 2; ++k) {
    if (g.h[k].n < 2) continue;
    for (m = 0; m < 2; ++m) {
      const int n = g.h[k].m[m].nc * g.h[k].m[m].nt;
      if (i < n) break;
      i -= n;
    }
    if (m < 2) break;
  }
  if (k == 2) return;
  const int n1 = g.h[k].m[1].nc * g.h[k].m[1].nt, others = m ? g.h[k].m[0].nc * g.h[k].m[0].nt : n1;
  const float *vec = g.h[k].m[1 - m].vec + r, *src = g.dst[k] + (size_t)(m ? i : i * n1) * g.R + r;
  const size_t step = (size_t)(m ? n1 : 1) * g.R;
  grid_dependency_wait();
  float v = 0.f;
  if (r < g.R)
#pragma unroll 8
    for (int o = y; o < others; o += 8) v = fmaf(src[o * step], vec[(size_t)o * g.R], v);
  red[y][x] = v;
  __syncthreads();
  if (y == 0 && r < g.R) {
#pragma unroll
    for (int w = 1; w < 8; ++w) v += red[w][x];
    g.grad[k][m][(size_t)i * g.R + r] = v;
  }
}

struct HalvesPlan {
  int na, a_size, b_size, atiles, btiles, splits, rblocks;
};
// CTAs of the pass: as many as are resident at once (fixed, as in contract_peel.cu: the order of the sums must not depend on the device)
constexpr int kSlots = 296;
HalvesPlan halves_plan(int L, const int* sizes, int R) {
  HalvesPlan best{};
  double least = 1e300;
  for (int na = L == 4 ? 2 : 1; na <= 2 && na < L; ++na) {
    HalvesPlan p{};
    p.na = na;
    p.a_size = p.b_size = 1;
    for (int k = 0; k < L; ++k) (k < p.na ? p.a_size : p.b_size) *= sizes[k];
    p.atiles = ceil_div(p.a_size, kHA);
    p.btiles = ceil_div(p.b_size, kHB);
    p.rblocks = ceil_div(R, kHR);
    p.splits = std::max(1, std::min(p.btiles, kSlots / (p.atiles * p.rblocks)));
    // three modes: the fewer tiles, of which the set-up of a CTA takes as long as one (12x16x16 -> 12x16x16 at R = 50: the first mode alone 123 us,
    // the first two 93; 16x10x6 -> 12x12x4 at R = 213, whose last mode fills a third of a tile, 55 and 125)
    const double tiles = (double)p.atiles * (p.btiles + p.splits);
    if (tiles < least) {
      least = tiles;
      best = p;
    }
  }
  return best;
}

}  // namespace

// Where this is faster than the peel.  2100 drawn layers of 4e4 to 1e7 entries and 4 to 256 ranks, kernel times over the peeled ones where the rule takes it,
// and where it does not:
//   three modes           2e6 entries, or 7e5 where the first is alone a; three tiles of b      0.45 to 1.03 (mean 0.73)   0.63 to 1.53 (0.95)
//   taps and two modes    1e5 entries, three tiles of b and 96 ranks at most                    0.57 to 0.96 (0.72)        0.59 to 1.55 (0.89)
//   four, taps and three  1e5 entries and three tiles of a, or 4e5 entries                      0.09 to 1.03 (0.63)        0.40 to 1.39 (0.85)
// A side of fewer tiles leaves most of an SM's time to the set-up; near these lines the times are 18 to 30 us.  (Two modes have at most 65536 entries.)
bool halves_take(int L, const int* sizes, int R, bool has_s) {
  const int mode = gemm_tc_mode();   // 0: no tensor products, 2: at every size
  if (L < 3 || L > 4 || !mode) return false;
  double entries = 1;
  for (int k = 0; k < L; ++k) entries *= sizes[k];
  if (entries >= 2147483647.0) return false;
  if (mode == 2) return true;
  const HalvesPlan p = halves_plan(L, sizes, R);
  if (L == 4) return entries >= 4e5 || (entries >= 1e5 && p.atiles >= 3);
  if (has_s) return entries >= 1e5 && p.btiles >= 3 && R <= 96;
  return entries >= (p.na == 1 ? 7e5 : 2e6) && p.btiles >= 3;
}

size_t halves_scratch_floats(int L, const int* sizes, int R) {
  const HalvesPlan p = halves_plan(L, sizes, R);
  return ((size_t)p.splits * p.a_size + (size_t)p.atiles * p.b_size + p.a_size + p.b_size) * R;
}

int halves_launch(int L, const PeelMode* modes, int R, const float* G, float* const* grads, float* scratch, cudaStream_t st) {
  int sizes[4];
  for (int k = 0; k < L; ++k) sizes[k] = modes[k].nc * modes[k].nt;
  const HalvesPlan p = halves_plan(L, sizes, R);
  HalvesGeom g{};
  HalvesSums s{};
  g.a.n = p.na; g.a.size = p.a_size;
  g.b.n = L - p.na; g.b.size = p.b_size;
  for (int k = 0; k < L; ++k) (k < p.na ? g.a.m[k] : g.b.m[k - p.na]) = modes[k];
  g.R = R; g.btiles = p.btiles; g.splits = p.splits; g.G = G;
  g.sa = scratch;
  g.sb = g.sa + (size_t)p.splits * p.a_size * R;
  float* sum = g.sb + (size_t)p.atiles * p.b_size * R;
  s.h[0] = g.a; s.h[1] = g.b; s.part[0] = g.sa; s.part[1] = g.sb; s.parts[0] = p.splits; s.parts[1] = p.atiles; s.R = R;
  int factors = 0;
  for (int k = 0; k < 2; ++k) {
    const int at = k ? p.na : 0;
    s.grad[k][0] = grads[at];
    if (s.h[k].n > 1) {
      s.grad[k][1] = grads[at + 1];
      s.dst[k] = sum;
      sum += (size_t)s.h[k].size * R;
      factors += sizes[at] + sizes[at + 1];
    } else {
      s.dst[k] = grads[at];
    }
  }
  // offsets of whole rows of C entries, of t digits of a and b, and of a's c digits are multiples of the last half's c entries
  int cb = 1;
  for (int k = 0; k < g.b.n; ++k) cb *= g.b.m[k].nc;
  const bool vec = !(cb & 3) && !(reinterpret_cast<uintptr_t>(G) & 15);
  const auto kernel = vec ? halves_kernel<true> : halves_kernel<false>;
  static std::atomic<int> set[2][64];
  B200CP_CUDA_OK(ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), set[vec], (int)kHalvesSmem));
  B200CP_CUDA_OK(launch_kernel(kernel, dim3(p.atiles, p.splits, p.rblocks), dim3(kHT), kHalvesSmem, st, true, g));
  B200CP_LAUNCH_OK("halves_kernel");
  const auto blocks = [&](int k) { return s.parts[k] > kManyParts ? s.h[k].size : ceil_div(s.h[k].size, 8); };
  s.blocks0 = blocks(0);
  B200CP_CUDA_OK(launch_kernel(halves_sum_kernel, dim3(s.blocks0 + blocks(1), p.rblocks), dim3(256), 0, st, true, s));
  B200CP_LAUNCH_OK("halves_sum_kernel");
  if (factors) {
    B200CP_CUDA_OK(launch_kernel(halves_factor_kernel, dim3(factors, p.rblocks), dim3(256), 0, st, true, s));
    B200CP_LAUNCH_OK("halves_factor_kernel");
  }
  return B200CP_OK;
}

// Reads (and clears) the status word; the caller has synchronised the device.
int halves_device_status(int* out) {
  int v = 0, zero = 0;
  B200CP_CUDA_OK(cudaMemcpyFromSymbol(&v, g_halves_status, sizeof(int)));
  if (v) B200CP_CUDA_OK(cudaMemcpyToSymbol(g_halves_status, &zero, sizeof(int)));
  *out = v;
  return B200CP_OK;
}

}  // namespace b200cp
