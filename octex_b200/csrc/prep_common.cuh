// Device pieces shared by the two projection kernels of a batch (project_tc.cu on the tensor cores,
// project_ord.cu in dimension order): the cell lookup of one (query, copy) and the sketch-space
// queries, which extra blocks of the same launch compute, so that a batch starts with one kernel.
#pragma once

#include "kernels.hpp"

#include "e8.cuh"

namespace octex_b200::kernels {

// A kernel launched with programmatic stream serialisation may start while the kernel before it in
// the stream still runs: it waits here before it reads or writes anything that kernel touches. The
// wait returns at once in a launch without the attribute.
__device__ __forceinline__ void wait_for_previous_kernel() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
/// Let the next kernel of the stream be scheduled as soon as blocks of this one leave room.
__device__ __forceinline__ void let_next_kernel_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ---- cell lookup -----------------------------------------------------------------------------------

/// Lanes that decode one (query, copy) together: one per block of eight coordinates where that is a
/// power of two. A lane of its own per (query, copy) would run its 650 instructions per spacing with
/// 32 coordinates and their intermediates in 128 registers, 16 warps to a multiprocessor and a
/// quarter of its issue slots used; a lane per block needs half the registers, and a lone query waits
/// for a quarter of the instructions.
template <int B>
constexpr int kGroup = (B & (B - 1)) == 0 ? B : 1;

/// The decodes off the usual path: coordinates of a million spacings and more, and blocks whose two
/// cosets are nearly as near (block_code_fast).
static __device__ __noinline__ unsigned long long block_code_rare(float v0, float v1, float v2, float v3, float v4,
                                                                  float v5, float v6, float v7, bool wild)
{
  const float v[8] = {v0, v1, v2, v3, v4, v5, v6, v7};
  return wild ? block_code(v) : block_code_tame(v);
}

/// Code of a block whose coordinates (scaled by inv) may be any; wild: one of them may be beyond
/// kTameLimit, margin: decode_margin of them.
__device__ __forceinline__ unsigned long long block_code_any(const f32_pair (&own)[4], float inv, float margin,
                                                             const unsigned long long* primes, bool wild)
{
  bool doubtful;
  unsigned long long hb = block_code_fast(own, inv, margin, primes, doubtful);
  if (wild || doubtful) {
    float v[8];
#pragma unroll
    for (int i = 0; i < 4; i++)
      unpack2(mul2(own[i], pack2(inv, inv)), v[2 * i], v[2 * i + 1]);
    hb = block_code_rare(v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], wild);
  }
  return hb;
}

/// The cell primes where block_code_fast reads them (8 words of shared memory, filled by the block).
__device__ __forceinline__ void fill_primes(unsigned long long* primes)
{
  if (threadIdx.x < 8) primes[threadIdx.x] = kCellPrimes[threadIdx.x];
}

/// Decodes the cell code of a (query, copy) spread over kGroup<B> lanes: lane `sub` of the group holds
/// blocks sub * kOwn .. of its coordinates. The chained sum h = (..(b0 G + b1) G + ..) + b_last of
/// cell_code is linear in the block codes, so every lane weighs its own part by its power of G and the
/// lanes add up (all modulo 2^64).
template <int B>
struct group_decoder {
  static constexpr int kOwn = B / kGroup<B>;
  f32_pair y[4 * kOwn];
  const unsigned long long* primes;
  unsigned long long weight;
  float reach;  // the largest magnitude of the coordinates (NaN: one of them is none)
  bool wild;

  __device__ __forceinline__ group_decoder(int sub, const unsigned long long* p) : primes(p)
  {
    weight = 1;
    for (int i = sub; i < kGroup<B> - 1; i++)
#pragma unroll
      for (int k = 0; k < kOwn; k++)
        weight *= kGolden;
  }
  /// Which of the decodes the coordinates need; call it when y is set.
  __device__ __forceinline__ void settle(float tame_y)
  {
    reach = 0.f;
#pragma unroll
    for (int i = 0; i < 4 * kOwn; i++) {
      float a, b;
      unpack2(y[i], a, b);
      reach = max_abs_nan(reach, max_abs_nan(a, b));
    }
    wild = !(reach < tame_y);
  }
  /// All lanes of the warp call it together.
  __device__ __forceinline__ long long code(float inv_f) const
  {
    unsigned long long h = 0;
    const float margin   = decode_margin(reach, inv_f);
#pragma unroll
    for (int j = 0; j < kOwn; j++) {
      f32_pair own[4];
#pragma unroll
      for (int i = 0; i < 4; i++)
        own[i] = y[4 * j + i];
      const unsigned long long hb = block_code_any(own, inv_f, margin, primes, wild);
      h = j == 0 ? hb : h * kGolden + hb;
    }
    if constexpr (kGroup<B> > 1) {
      h *= weight;
#pragma unroll
      for (int o = 1; o < kGroup<B>; o <<= 1)
        h += __shfl_xor_sync(0xffffffffu, h, o);
    }
    return finish_code(h);
  }
};

/// Row of the cell of a code in a level's table, -1 when there is no such cell: slot by slot from the
/// home bucket on, every tag that fits confirmed at once. For inspection, and for the lookups a search
/// could not settle in passing (a full bucket, a tag two codes share). All arguments in registers.
static __device__ __noinline__ int lookup_exact(const cell_slot* table, const long long* keys, unsigned mask, long long code)
{
  unsigned s = cell_home(code, mask);
  for (unsigned probe = 0; probe <= mask; probe++) {
    const int2 slot = __ldg(reinterpret_cast<const int2*>(table + s));
    if (slot.y < 0) return -1;  // an empty slot ends the run
    if (slot.x == cell_tag(code) && keys[slot.y] == code) return slot.y;
    s = (s + 1) & mask;
  }
  return -1;
}

/// What a lookup found in its home bucket.
constexpr int kNoCell  = -1;  // no such cell
constexpr int kNotSure = -2;  // a bucket full of other cells: lookup_exact says

/// A lane group's lookup of a code: a lane of a group of four holds one slot of the home bucket (a lane
/// of a group of two two, a lane alone all four, of the eight lanes of a group the last four none).
template <int kG>
struct group_lookup {
  static constexpr int kHold = kG >= 4 ? 1 : 4 / kG;
  long long code = 0;
  int2 slot[kHold];
  bool pending = false;

  __device__ __forceinline__ void request(const tc_lookup& look, const cell_level& lv, long long c, int sub)
  {
    code                  = c;
    const cell_slot* home = look.table + lv.off + cell_home(c, static_cast<unsigned>(lv.mask)) + (sub & (4 / kHold - 1)) * kHold;
    if constexpr (kHold == 1) {
      slot[0] = __ldg(reinterpret_cast<const int2*>(home));
    } else {
#pragma unroll
      for (int i = 0; i < kHold; i += 2) {
        const int4 two = __ldg(reinterpret_cast<const int4*>(home + i));
        slot[i]        = make_int2(two.x, two.y);
        slot[i + 1]    = make_int2(two.z, two.w);
      }
    }
    pending = true;
  }
  /// Row of the cell, kNoCell or kNotSure, for the groups with a lookup pending; kNoCell for the others.
  /// The tag is all that has been compared. All lanes of the warp call it together.
  __device__ __forceinline__ int resolve()
  {
    int row     = -1;
    bool vacant = false;
#pragma unroll
    for (int i = 0; i < kHold; i++) {
      if (slot[i].x == cell_tag(code) && slot[i].y >= 0) row = slot[i].y;
      vacant = vacant || slot[i].y < 0;
    }
    if constexpr (kG > 1) {
      const int lane       = threadIdx.x & 31;
      const unsigned group = ((1u << kG) - 1u) << (lane & ~(kG - 1));
      const unsigned match = __ballot_sync(0xffffffffu, pending && row >= 0) & group;
      vacant               = (__ballot_sync(0xffffffffu, vacant) & group) != 0;
      row                  = __shfl_sync(0xffffffffu, row, match != 0 ? __ffs(match) - 1 : lane);
      if (match == 0) row = -1;
    }
    const int out = !pending ? kNoCell : row >= 0 ? row : vacant ? kNoCell : kNotSure;
    pending       = false;
    return out;
  }
};

/// First list entry of the cell, -1 when there is none, from what resolve() said: a tag that fits is
/// confirmed against the whole code.
__device__ __forceinline__ int lookup_settle(const tc_lookup& look, const cell_level& lv, long long code, int row)
{
  if (row == kNoCell) return -1;
  if (row < 0 || __ldg(look.keys + lv.keys + row) != code)
    row = lookup_exact(look.table + lv.off, look.keys + lv.keys, static_cast<unsigned>(lv.mask), code);
  return row < 0 ? -1 : (lv.base + row) * look.list_len;
}

/// Segments of the pairs (query, copy) of a block: pair p is local row p / kC, local copy p % kC, and
/// fetch(p, sub, y) brings the coordinates of lane sub's blocks; lv [kC * L] are the levels of the
/// block's copies and primes fill_primes' (both shared memory). For every pair the finest level whose cell holds a list
/// (search_kernels.cuh:100-126 of the reference). A lane group takes a pair and goes through the
/// levels; the bucket of a level is requested as soon as its code is known and looked at after the
/// next level has been decoded, so its latency hides behind that decode; once a level hits, the
/// coarser ones are not decoded at all. No code goes to memory. All threads of the block call it.
template <int B, int kC, typename Fetch>
__device__ __forceinline__ void lookup_pairs(const tc_lookup& look, Fetch fetch, int pairs, float tame_y,
                                             const float* inv_f, const cell_level* lv,
                                             const unsigned long long* primes, int L, int64_t row0, int c0, int Cg)
{
  constexpr int kG = kGroup<B>;
  const int sub    = threadIdx.x % kG;
  group_decoder<B> dec(sub, primes);
  for (int p0 = (threadIdx.x / 32) * (32 / kG); p0 < pairs; p0 += blockDim.x / kG) {
    const int p = p0 + (threadIdx.x % 32) / kG;
    const int c = c0 + p % kC;
    const bool live = p < pairs && c < Cg;
    fetch(min(p, pairs - 1), sub, dec.y);
    dec.settle(tame_y);
    int first = -1, asked = 0;
    group_lookup<kG> ask;
    int tried = 0;  // levels, a bucket of four slots each
    auto answer = [&] {
      const bool was = ask.pending;
      const int row  = ask.resolve();
      if (!was) return;
      tried++;
      first = lookup_settle(look, lv[(p % kC) * L + asked], ask.code, row);
    };
    for (int j = 0; j < L; j++) {
      const bool want = live && first < 0 && lv[(p % kC) * L + j].mask >= 0;
      if (!__any_sync(0xffffffffu, want)) {
        if (!__any_sync(0xffffffffu, live && first < 0)) break;
        continue;
      }
      const long long h = dec.code(inv_f[j]);
      answer();
      if (want && first < 0) {
        asked = j;
        ask.request(look, lv[(p % kC) * L + j], h, sub);
      }
    }
    answer();
    if (live && sub == 0) {
      const int64_t row      = row0 + p / kC;
      look.seg[row * Cg + c] = first >= 0 ? make_int2(first, look.lr) : make_int2(0, 0);
      if (look.stats != nullptr) {
        atomicAdd(reinterpret_cast<unsigned long long*>(look.stats + row * 8), static_cast<unsigned long long>(tried));
        atomicAdd(reinterpret_cast<unsigned long long*>(look.stats + row * 8 + 1), static_cast<unsigned long long>(4 * tried));
      }
    }
  }
}

/// The segment of one (query, copy) by one thread with all of its coordinates (4 B pairs): the form for
/// large batches, where the instructions of a step count and not how long a warp takes for it. A lane
/// per block repeats what follows the decode (final mixing, lookup) in every lane of the group. reach:
/// the largest magnitude of the coordinates; wild: it is beyond the short decodes. All lanes of the
/// warp call it together; lv [L] are the levels of the copy.
template <int B>
__device__ __forceinline__ void lookup_alone(const tc_lookup& look, const f32_pair (&y)[4 * B], bool live, float reach,
                                             bool wild, const float* inv_f, const cell_level* lv,
                                             const unsigned long long* primes, int L, int64_t row, int c, int Cg)
{
  int first = -1, asked = 0;
  group_lookup<1> ask;
  int tried = 0;  // levels, a bucket of four slots each
  auto answer = [&] {
    if (!ask.pending) return;
    tried++;
    first = lookup_settle(look, lv[asked], ask.code, ask.resolve());
  };
  for (int j = 0; j < L; j++) {
    const bool want = live && first < 0 && lv[j].mask >= 0;
    if (!__any_sync(0xffffffffu, want)) {
      if (!__any_sync(0xffffffffu, live && first < 0)) break;
      continue;
    }
    unsigned long long h = 0;
    const float margin   = decode_margin(reach, inv_f[j]);
#pragma unroll
    for (int b = 0; b < B; b++) {
      f32_pair own[4];
#pragma unroll
      for (int i = 0; i < 4; i++)
        own[i] = y[4 * b + i];
      h = h * kGolden + block_code_any(own, inv_f[j], margin, primes, wild);
    }
    const long long code = finish_code(h);
    answer();
    if (want && first < 0) {
      asked = j;
      ask.request(look, lv[j], code, 0);
    }
  }
  answer();
  if (!live) return;
  look.seg[row * Cg + c] = first >= 0 ? make_int2(first, look.lr) : make_int2(0, 0);
  if (look.stats != nullptr) {
    atomicAdd(reinterpret_cast<unsigned long long*>(look.stats + row * 8), static_cast<unsigned long long>(tried));
    atomicAdd(reinterpret_cast<unsigned long long*>(look.stats + row * 8 + 1), static_cast<unsigned long long>(4 * tried));
  }
}

/// The same for a block with so few pairs that most lane groups would have none: every (pair, level)
/// is worked on by a group of its own, all at once, and the finest hit is taken: the same answer, some
/// levels decoded for nothing. best [pairs] and hit [pairs * L] are scratch in shared memory; needs
/// look.stats == nullptr. All threads of the block call it.
template <int B>
__host__ __device__ constexpr bool spread_pays(int pairs, int L)
{
  return L > 1 && pairs * L * kGroup<B> <= 512;
}
template <int B, int kC, typename Fetch>
__device__ __forceinline__ void lookup_spread(const tc_lookup& look, Fetch fetch, int* best, int* hit, int pairs,
                                              float tame_y, const float* inv_f, const cell_level* lv,
                                              const unsigned long long* primes, int L, int64_t row0, int c0, int Cg)
{
  constexpr int kG = kGroup<B>;
  const int sub    = threadIdx.x % kG;
  for (int p = threadIdx.x; p < pairs; p += blockDim.x)
    best[p] = L;
  __syncthreads();
  group_decoder<B> dec(sub, primes);
  for (int i0 = (threadIdx.x / 32) * (32 / kG); i0 < pairs * L; i0 += blockDim.x / kG) {
    const int item  = i0 + (threadIdx.x % 32) / kG;
    const bool live = item < pairs * L;
    const int j = live ? item / pairs : 0, p = live ? item - j * pairs : 0;
    const cell_level level = lv[(p % kC) * L + j];
    fetch(p, sub, dec.y);
    dec.settle(tame_y);
    const long long h = dec.code(inv_f[j]);
    group_lookup<kG> ask;
    if (live && c0 + p % kC < Cg && level.mask >= 0) ask.request(look, level, h, sub);
    const bool was    = ask.pending;
    const int row     = ask.resolve();
    const int first   = was ? lookup_settle(look, level, h, row) : -1;
    if (first >= 0 && sub == 0) {
      hit[item] = first;
      atomicMin(&best[p], j);
    }
  }
  __syncthreads();
  for (int p = threadIdx.x; p < pairs; p += blockDim.x) {
    const int c = c0 + p % kC, j = best[p];
    if (c < Cg) look.seg[(row0 + p / kC) * Cg + c] = j < L ? make_int2(hit[j * pairs + p], look.lr) : make_int2(0, 0);
  }
}

// ---- sketch-space queries -----------------------------------------------------------------------------

// qs = (q - mean) @ basis in fp32 (search.cu:321-341 of the reference), each (query, coordinate) sum
// running over the dimensions in order with one fused multiply-add per dimension. A block of 256
// threads takes a tile of queries x coordinates, a thread eight queries by kC coordinates of it. Both
// operands pass through shared memory in steps of dimensions, the next step's loads in flight while a
// step is summed: a lone query is a serial chain of D multiply-adds, and this keeps memory latency out
// of it (960 dimensions x 128 coordinates x 999 queries took 166 us as a kernel of its own that read
// the basis in the sum; here it runs beside the projection). Two tiles: 64 x 32, one coordinate per
// thread, for small batches, where the number of blocks counts, and 128 x 64, four coordinates per
// thread, for large ones, where three shared-memory reads then serve 32 multiply-adds instead of
// eight (10 000 queries x 128 dimensions x 64 coordinates: 20 us of the projection's time with the
// small tile).
template <int kC>
struct sketch_tile {
  static constexpr int kCols = kC == 1 ? 32 : 16 * kC;
  static constexpr int kRows = 256 / (kCols / kC) * 8;
  static constexpr int kDims = kC == 1 ? 64 : 32;
  static constexpr int kLd   = kRows + 4;
  static constexpr int kWords = kDims * (kLd + kCols);  // floats of shared memory
};

template <int kC>
__host__ __device__ inline int sketch_blocks(const sketch_job& j)
{
  using T = sketch_tile<kC>;
  return ((j.m + T::kRows - 1) / T::kRows) * ((j.S + T::kCols - 1) / T::kCols);
}

template <int kC>
__device__ __forceinline__ void sketch_block(const sketch_job& j, int block, float* smem)
{
  using T          = sketch_tile<kC>;
  float* xs        = smem;                      // [dims][rows + 4]: centred queries
  float* bs        = smem + T::kDims * T::kLd;  // [dims][coordinates]
  const int slabs  = (j.S + T::kCols - 1) / T::kCols;
  const int col0   = (block % slabs) * T::kCols;
  const int row0   = (block / slabs) * T::kRows;
  const int rows   = min(T::kRows, j.m - row0);
  const int col    = threadIdx.x % (T::kCols / kC) * kC, rg = threadIdx.x / (T::kCols / kC);
  const bool keeps = col0 == 0 && j.keep != nullptr;
  constexpr int kX = T::kRows * T::kDims / 256, kB = T::kCols * T::kDims / 256;
  float x[kX], b[kB];
  auto fetch = [&](int d0) {
#pragma unroll
    for (int u = 0; u < kX; u++) {
      const int i = threadIdx.x + u * 256, r = i / T::kDims, d = d0 + i % T::kDims;
      x[u] = r < rows && d < j.D ? __ldg(j.q + static_cast<int64_t>(row0 + r) * j.D + d) : 0.f;
    }
#pragma unroll
    for (int u = 0; u < kB; u++) {
      const int i = threadIdx.x + u * 256, d = d0 + i / T::kCols, c = col0 + i % T::kCols;
      b[u] = d < j.D && c < j.S ? __ldg(j.basis + static_cast<int64_t>(d) * j.S + c) : 0.f;
    }
  };
  float acc[8][kC];
#pragma unroll
  for (int r = 0; r < 8; r++)
#pragma unroll
    for (int k = 0; k < kC; k++)
      acc[r][k] = 0.f;
  fetch(0);
  for (int d0 = 0; d0 < j.D; d0 += T::kDims) {
    const int mine = threadIdx.x % T::kDims;  // every x of a thread is of the same dimension
    const float mu = d0 + mine < j.D ? __ldg(j.mean + d0 + mine) : 0.f;
#pragma unroll
    for (int u = 0; u < kX; u++) {
      const int r = (threadIdx.x + u * 256) / T::kDims;
      if (keeps && r < rows && d0 + mine < j.D) j.keep[static_cast<int64_t>(row0 + r) * j.D + d0 + mine] = x[u];
      if (r < rows) xs[mine * T::kLd + r] = __fsub_rn(x[u], mu);
    }
#pragma unroll
    for (int u = 0; u < kB; u++)
      bs[threadIdx.x + u * 256] = b[u];
    __syncthreads();
    if (d0 + T::kDims < j.D) fetch(d0 + T::kDims);
    if (8 * rg < rows) {
      const int dd = min(T::kDims, j.D - d0);
#pragma unroll 4
      for (int d = 0; d < dd; d++) {
        const float4 x0   = *reinterpret_cast<const float4*>(xs + d * T::kLd + 8 * rg);
        const float4 x1   = *reinterpret_cast<const float4*>(xs + d * T::kLd + 8 * rg + 4);
        const float xv[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
        float w[kC];
        if constexpr (kC == 4) {
          const float4 w4 = *reinterpret_cast<const float4*>(bs + d * T::kCols + col);
          w[0] = w4.x, w[1] = w4.y, w[2] = w4.z, w[3] = w4.w;
        } else {
          w[0] = bs[d * T::kCols + col];
        }
#pragma unroll
        for (int r = 0; r < 8; r++)
#pragma unroll
          for (int k = 0; k < kC; k++)
            acc[r][k] = __fmaf_rn(xv[r], w[k], acc[r][k]);
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int r = 0; r < 8; r++)
#pragma unroll
    for (int k = 0; k < kC; k++)
      if (8 * rg + r < rows && col0 + col + k < j.S)
        j.qs[static_cast<int64_t>(row0 + 8 * rg + r) * j.S + col0 + col + k] = acc[r][k];
}

}  // namespace octex_b200::kernels
