// Projection of a query batch on all copies with the E8 decode and the cell lookup in the epilogue
// (sm_100a only):
//   acc[m, Cg*32] = half(q - mean)[m, K] . ut[Cg*32, K]^T   tcgen05.mma, fp16 in, fp32 accumulators in TMEM
//   y = half(acc + shift)                                   what the reference's GEMM writes out
//   seg[q, c] = first list entry of the finest populated cell among those of y[q, c*32 .. c*32+32)
//
// Answers center_kernel, the cuBLASLt call and probe_kernel of the reference (hpdic/octex,
// cpp/src/neighbors/octex/search.cu:139-168, 303-320: fp16 operands, fp32 accumulate, fp16 bias
// epilogue, fp16 output; detail/search_kernels.cuh:57-69,100-126). Neither the centred queries nor
// the projected coordinates nor the codes go to memory: the block centres and rounds its queries
// while it writes the operand tile; a thread of the epilogue reads the 32
// accumulator columns of one copy from TMEM (tcgen05.ld 32x32b.x32 hands a lane exactly one copy),
// rounds them to fp16 and hands them through shared memory to groups of four lanes, one block of
// eight coordinates each, which decode the populated spacings and look their cells up.
//
// A tile is 128 queries (fewer in the spread form) x 64 coordinates (two copies), a block 256 threads. The projections come in by
// TMA (cp.async.bulk.tensor, no cluster forms), 64 rows x 64 halves (128 bytes, the swizzle span) a
// step; the queries are read as fp32 by all threads and written in the same swizzled layout; one
// thread issues the copies and the MMAs; every wait on an mbarrier is bounded and a wait that runs out
// sets an error word, lets the copies in flight land, frees the block's TMEM and returns. The
// sketch-space queries (sketch_block), which the rounds need and the projection does not, are made by
// blocks of the same launch.
//
// What bounds it: instruction issue of the decode (51 % of the slots at 16 warps a multiprocessor, 8.0 k warp
// instructions a query where the decode that repairs both cosets took 12.2 k) and the random sectors of
// the lookup. Two forms (tc_mode). 10 000 queries x 64 copies x 128 dimensions: 163 us in the bulk form
// with the sketch-space queries in it, against 188 + 27 us for a kernel that decoded two copies per
// thread after a 128-column tile and a centring kernel before it. One query: 10 us in the spread form
// against 24 + 11.

#include "kernels.hpp"

#include "prep_common.cuh"
#include "tc_common.cuh"

#include <algorithm>
#include <cstring>

namespace octex_b200::kernels {

namespace {

constexpr int kTileM    = 128;  // queries per tile = TMEM lanes
constexpr int kCopies   = 2;    // copies per tile
constexpr int kTileN    = 32 * kCopies;
constexpr int kStages   = 2;
constexpr int kThreads  = 256;  // two warps per TMEM lane quarter, one copy each
constexpr int kTmemCols = 2 * kTileN;  // two fp32 accumulators
constexpr int kBulkBlocks   = 2;  // blocks per SM of the form for large batches: 128 registers per thread
constexpr int kSpreadBlocks = 3;  // and of the form for others: 80
constexpr uint32_t kBBytes = kTileN * kTileK * 2;

struct __align__(1024) tc_smem {
  __half a[kStages][kTileM * kTileK];  // also the sketch blocks' staging and, once the MMAs are done,
  __half b[2 * kStages][kTileN * kTileK];  // the fp16 coordinates (a[0]) and the scratch of lookup_spread (a[1])
  uint64_t full[2 * kStages];
  uint64_t empty[kStages];
  uint64_t done;
  uint32_t tmem_base;
  int failed;
  float shift[2][kTileN];
  float inv_f[16];
  cell_level lv[2][kCopies * 16];
  unsigned long long primes[8];
};
// only a: TMA writes b, and nothing orders it after what threads did there
static_assert(sizeof(tc_smem::a) >= sizeof(float) * (sketch_tile<1>::kWords > sketch_tile<4>::kWords ? sketch_tile<1>::kWords
                                                                                                      : sketch_tile<4>::kWords),
              "staging of the sketch blocks");

/// Centred fp16 queries q[0, rows) (128 at most) x dimensions [d0, d0 + 64) into an operand tile with the
/// 128-byte swizzle (16-byte chunk c of row r at chunk c ^ (r % 8)). Rows beyond are left
/// as they are: an accumulator row depends on its own operand row only.
template <bool kVec>
__device__ __forceinline__ void fill_queries(__half* tile, const float* __restrict__ q, const float* __restrict__ mean,
                                             int rows, int D, int d0)
{
  const int part = threadIdx.x & 15, d = d0 + 4 * part;
  float mu[4];
#pragma unroll
  for (int i = 0; i < 4; i++)
    mu[i] = d + i < D ? __ldg(mean + d + i) : 0.f;
  float v[8][4];
#pragma unroll
  for (int u = 0; u < 8; u++) {
    const int r = (threadIdx.x >> 4) + 16 * u;
#pragma unroll
    for (int i = 0; i < 4; i++)
      v[u][i] = mu[i];
    if (r < rows) {
      const float* src = q + r * D + d;  // (32 bits hold 128 queries of 16 million dimensions)
      if constexpr (kVec) {
        if (d < D) {
          const float4 x = __ldg(reinterpret_cast<const float4*>(src));
          v[u][0] = x.x, v[u][1] = x.y, v[u][2] = x.z, v[u][3] = x.w;
        }
      } else {
#pragma unroll
        for (int i = 0; i < 4; i++)
          if (d + i < D) v[u][i] = __ldg(src + i);
      }
    }
  }
#pragma unroll
  for (int u = 0; u < 8; u++) {
    const int r = (threadIdx.x >> 4) + 16 * u;
    if (r >= rows) continue;
    __half h[4];
#pragma unroll
    for (int i = 0; i < 4; i++)
      h[i] = __float2half_rn(__fsub_rn(v[u][i], mu[i]));  // zero beyond the dimension
    uint2 w;
    w.x = static_cast<uint32_t>(__half_as_ushort(h[0])) | static_cast<uint32_t>(__half_as_ushort(h[1])) << 16;
    w.y = static_cast<uint32_t>(__half_as_ushort(h[2])) | static_cast<uint32_t>(__half_as_ushort(h[3])) << 16;
    *reinterpret_cast<uint2*>(reinterpret_cast<char*>(tile) + r * 128 + (((part >> 1) ^ (r & 7)) << 4) + (part & 1) * 8) = w;
  }
}

// kTaps: codes of every level and the coordinates are written out instead of looking the cells up.
// kSpread: a batch of few tiles, one per block, decoded by a lane per block of coordinates
// (group_decoder) after the blocks of the sketch-space queries. kBulk: a block for every place on the
// GPU goes through its share of the tiles, a thread per (query, copy), the next tile's projections on
// their way during the decode; the queries of a tile stay in shared memory from tile to tile when they
// fit its two stages. Which: project_decode_tc.
enum class tc_mode { taps, spread, bulk };
template <bool kVec, tc_mode kMode>
__global__ void __launch_bounds__(kThreads, kMode == tc_mode::taps ? 1 : kMode == tc_mode::spread ? kSpreadBlocks : kBulkBlocks)
  project_decode_tc_kernel(
  const __grid_constant__ CUtensorMap map_b,
  const sketch_job job,
  int sk_blocks,
  int rows,
  int Cg,
  int L,
  int nkb,
  const __half* __restrict__ shift,
  const float* __restrict__ inv_f,
  float tame_y,
  long long* __restrict__ codes,
  __half* __restrict__ Yout,
  const tc_lookup look,
  int* __restrict__ error)
{
  extern __shared__ unsigned char raw[];
  tc_smem& sm = *reinterpret_cast<tc_smem*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~uintptr_t{1023});
  let_next_kernel_start();
  if constexpr (kMode == tc_mode::bulk) {
    for (int b = blockIdx.x; b < sk_blocks; b += gridDim.x)
      sketch_block<4>(job, b, reinterpret_cast<float*>(&sm));
    __syncthreads();
  } else if (static_cast<int>(blockIdx.x) < sk_blocks) {
    sketch_block<1>(job, blockIdx.x, reinterpret_cast<float*>(&sm));
    return;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m = job.m, D = job.D;
  const int N       = Cg * 32;
  const int tiles_n = (Cg + kCopies - 1) / kCopies;
  const int tiles   = tiles_n * ((m + rows - 1) / rows);
  // the block's tiles, the copies of a tile of queries side by side
  int tile = blockIdx.x - sk_blocks, last = tile + 1;
  if constexpr (kMode == tc_mode::bulk) {
    tile = static_cast<int>(int64_t{tiles} * blockIdx.x / gridDim.x);
    last = static_cast<int>(int64_t{tiles} * (blockIdx.x + 1) / gridDim.x);
  }

  // Operands of few dimensions fit the stages whole: then the accumulators are double buffered, the
  // tensor cores work on the next tile during the decode of this one, and the projections of the one
  // after it come in (stages 2 set and 2 set + 1 for tiles of either parity).
  const bool ahead = kMode == tc_mode::bulk && nkb <= kStages;
  auto load_projections = [&](int of_tile, int kb, int set) {
    const int s = kStages * set + kb % kStages;
    mbar_expect_tx(&sm.full[s], kBBytes);
    tma_load_2d(sm.b[s], &map_b, kb * kTileK, (of_tile % tiles_n) * kTileN, &sm.full[s]);
  };
  // what the epilogue of a tile needs besides the accumulators
  auto fetch_levels = [&](int of_tile, int set) {
    const int tile_n = of_tile % tiles_n;
    if (threadIdx.x < kTileN) {
      const int col              = tile_n * kTileN + threadIdx.x;
      sm.shift[set][threadIdx.x] = col < N ? __half2float(shift[col]) : 0.f;
    }
    if (kMode != tc_mode::taps && threadIdx.x < kCopies * L)
      sm.lv[set][threadIdx.x] = tile_n * kCopies + threadIdx.x / L < Cg ? look.levels[tile_n * kCopies * L + threadIdx.x] : cell_level{0, 0, -1, 0};
  };
  if (threadIdx.x == 0) {
    for (int s = 0; s < 2 * kStages; s++)
      mbar_init(&sm.full[s], 1);
    for (int s = 0; s < kStages; s++)
      mbar_init(&sm.empty[s], 1);
    mbar_init(&sm.done, 1);
    sm.failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (int t = tile; t < min(last, tile + (ahead ? 2 : 1)); t++)
      for (int kb = 0; kb < min(nkb, kStages); kb++)
        load_projections(t, kb, t - tile);
  }
  if (threadIdx.x < L) sm.inv_f[threadIdx.x] = inv_f[threadIdx.x];
  fill_primes(sm.primes);
  if (tile < last) fetch_levels(tile, 0);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(&sm.tmem_base)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = sm.tmem_base;

  // instruction descriptor: D fp32, A and B fp16, both K-major, N = 64, M = 128
  constexpr uint32_t idesc = (1u << 4) | (static_cast<uint32_t>(kTileN >> 3) << 17) |
                             (static_cast<uint32_t>(kTileM >> 4) << 24);
  uint32_t full_phase = 0, empty_phase = 0, done_phase = 0;  // a bit per stage; of one tile after the other
  // by one thread: the MMAs of a 64-dimension step, once its projections are there
  auto step = [&](int kb, int set) {
    const int s = kStages * set + kb % kStages;
    if (!mbar_wait(&sm.full[s], (full_phase >> s) & 1u)) return false;
    full_phase ^= 1u << s;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint64_t da = umma_desc(sm.a[kb % kStages]), db = umma_desc(sm.b[s]);
#pragma unroll
    for (int k = 0; k < kTileK / 16; k++)  // 16 halves = 32 bytes = 2 descriptor units per step
      umma_f16(tmem + static_cast<uint32_t>(set * kTileN), da + 2 * k, db + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
    return true;
  };
  // all threads: the queries of a tile into the operand stages, when they fit whole
  auto fill_all = [&](int tile_m) {
    for (int kb = 0; kb < nkb; kb++)
      fill_queries<kVec>(sm.a[kb], job.q + static_cast<int64_t>(tile_m) * rows * D, job.mean, min(rows, m - tile_m * rows), D, kb * kTileK);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the tensor cores read what was just written
    __syncthreads();
  };
  bool ready = true;  // of every thread; one that gave up stops taking part in the waits, not in the barriers
  int set    = 0;
  if (ahead && tile < last) {
    fill_all(tile / tiles_n);
    if (threadIdx.x == 0) {
      for (int kb = 0; kb < nkb; kb++)
        ready = ready && step(kb, 0);
      if (ready)
        umma_commit(&sm.done);
      else
        sm.failed = 1;
    }
    __syncwarp();
  }
  for (; tile < last; tile++, set ^= ahead ? 1 : 0) {
    const int tile_n = tile % tiles_n, tile_m = tile / tiles_n;
    // The tile's queries, once: a row's place worked out for every 64 dimensions from the tile's number took one query of 960
    // dimensions 89.9 us a search instead of 89.3, its first and last row kept instead 40 queries 99.5 instead of 98.4.
    const float* const tile_q = job.q + static_cast<int64_t>(tile_m) * rows * D;
    const int tile_rows       = min(rows, m - tile_m * rows);
    if (ahead) {
      ready = ready && mbar_wait(&sm.done, done_phase, &sm.failed);
      if (!ready) sm.failed = 1;
      // every thread has read the other accumulator and the other levels: the tile before is over
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncthreads();
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (tile + 1 < last) {
        fetch_levels(tile + 1, set ^ 1);
        if ((tile + 1) / tiles_n != tile_m) fill_all((tile + 1) / tiles_n);
        if (threadIdx.x == 0 && ready) {
          for (int kb = 0; kb < nkb; kb++)
            ready = ready && step(kb, set ^ 1);
          if (ready) {
            umma_commit(&sm.done);
            if (tile + 2 < last)
              for (int kb = 0; kb < nkb; kb++)
                load_projections(tile + 2, kb, set);
          } else {
            sm.failed = 1;
          }
        }
      }
    } else {
      if (kMode == tc_mode::bulk) {
        // every thread is done with what it reads of these from the tile before
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        fetch_levels(tile, 0);
      }
      for (int kb = 0; kb < nkb; kb++) {
        const int s = kb % kStages;
        if (kb >= kStages) {
          // the MMAs that read this stage are done
          ready = ready && mbar_wait(&sm.empty[s], (empty_phase >> s) & 1u, &sm.failed);
          empty_phase ^= 1u << s;
          if (!ready) sm.failed = 1;
          if (ready && threadIdx.x == 0) load_projections(tile, kb, 0);
        }
        if (ready) fill_queries<kVec>(sm.a[s], tile_q, job.mean, tile_rows, D, kb * kTileK);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (threadIdx.x == 0 && ready) {
          ready = step(kb, 0);
          if (ready) {
            if (kb + kStages < nkb) umma_commit(&sm.empty[s]);
            if (kb + 1 == nkb) umma_commit(&sm.done);
          } else {
            sm.failed = 1;
          }
        }
      }
      __syncwarp();
      // everybody waits for the accumulators (or for the failure mark a thread that gave up leaves)
      ready = ready && mbar_wait(&sm.done, done_phase, &sm.failed);
      // the stages are free: the projections of the next tile come in behind the decode of this one
      if (ready && threadIdx.x == 0 && tile + 1 < last)
        for (int kb = 0; kb < min(nkb, kStages); kb++)
          load_projections(tile + 1, kb, 0);
    }
    done_phase ^= 1u;
    if (!ready && threadIdx.x == 0) atomicExch(error, 1);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncwarp();

    // warp w reads TMEM lanes 32 (w % 4) .. + 31; warps 0-3 take the first copy of the tile, 4-7 the second
    const int quarter = warp & 3, cc = warp >> 2;
    const int row = tile_m * rows + quarter * 32 + lane;  // (a tile has all 128 in the forms that use it)
    const int c   = tile_n * kCopies + cc;
    uint32_t r[32];
    const uint32_t taddr = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + static_cast<uint32_t>(set * kTileN + cc * 32);
    asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
        "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]),
        "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]),
        "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    if constexpr (kMode == tc_mode::taps) {
      if (ready && row < m && c < Cg) {
        float y[32];
        __align__(16) __half yh[32];
        bool wild = false;  // a coordinate too large for the short decode (or not a number)
  #pragma unroll
        for (int i = 0; i < 32; i++) {
          yh[i] = __float2half_rn(__fadd_rn(__uint_as_float(r[i]), sm.shift[set][cc * 32 + i]));
          y[i]  = __half2float(yh[i]);
          wild  = wild || !(fabsf(y[i]) < tame_y);
        }
        uint4* dst = reinterpret_cast<uint4*>(Yout + static_cast<int64_t>(row) * N + c * 32);
  #pragma unroll
        for (int i = 0; i < 4; i++)
          dst[i] = *reinterpret_cast<const uint4*>(&yh[8 * i]);
        long long* out = codes + (static_cast<int64_t>(row) * Cg + c) * L;
        for (int j = 0; j < L; j++)
          out[j] = wild ? cell_code<4>(y, sm.inv_f[j]) : cell_code_tame<4>(y, sm.inv_f[j]);
      }
    } else if constexpr (kMode == tc_mode::bulk) {
      f32_pair y[16];
      float reach = 0.f;  // the largest magnitude (NaN: a coordinate is not a number)
  #pragma unroll
      for (int i = 0; i < 16; i++) {
        const float2 sh = *reinterpret_cast<const float2*>(sm.shift[set] + cc * 32 + 2 * i);
        const float a   = __half2float(__float2half_rn(__fadd_rn(__uint_as_float(r[2 * i]), sh.x)));
        const float b   = __half2float(__float2half_rn(__fadd_rn(__uint_as_float(r[2 * i + 1]), sh.y)));
        reach           = max_abs_nan(reach, max_abs_nan(a, b));
        y[i]            = pack2(a, b);
      }
      // a row beyond the batch holds anything: it goes through the motions of the short decode
      const bool live = ready && row < m && c < Cg;
      lookup_alone<4>(look, y, live, live ? reach : 0.f, live && !(reach < tame_y), sm.inv_f, sm.lv[set] + cc * L, sm.primes, L, row, c, Cg);
    } else {
      // The coordinates change hands through shared memory: row e of the tile is a line of 128 bytes,
      // chunk 4 cc + j (16 bytes) holds block j of copy cc, at chunk ^ (e % 8) so that neither side has
      // bank conflicts. Every thread has left the wait above, so the MMAs that read the tiles are over.
      char* ys             = reinterpret_cast<char*>(sm.a[0]);
      const bool all_ready = __syncthreads_and(ready);
      const int e = quarter * 32 + lane;
  #pragma unroll
      for (int j = 0; j < 4; j++) {
        uint32_t h2[4];
  #pragma unroll
        for (int i = 0; i < 4; i++) {
          const float2 sh = *reinterpret_cast<const float2*>(sm.shift[set] + cc * 32 + 8 * j + 2 * i);
          const __half2 h = __halves2half2(__float2half_rn(__fadd_rn(__uint_as_float(r[8 * j + 2 * i]), sh.x)),
                                           __float2half_rn(__fadd_rn(__uint_as_float(r[8 * j + 2 * i + 1]), sh.y)));
          h2[i]           = *reinterpret_cast<const uint32_t*>(&h);
        }
        *reinterpret_cast<uint4*>(ys + e * 128 + (((4 * cc + j) ^ (e & 7)) << 4)) = make_uint4(h2[0], h2[1], h2[2], h2[3]);
      }
      __syncthreads();
      auto coordinates = [&](int p, int sub, f32_pair(&y)[4]) {
        const int at  = p / kCopies;
        const uint4 v = *reinterpret_cast<const uint4*>(ys + at * 128 + (((4 * (p % kCopies) + sub) ^ (at & 7)) << 4));
        const uint32_t h2[4] = {v.x, v.y, v.z, v.w};
  #pragma unroll
        for (int i = 0; i < 4; i++) {
          const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h2[i]));
          y[i]           = pack2(f.x, f.y);
        }
      };
      const int pairs    = min(rows, m - tile_m * rows) * kCopies;
      const int64_t row0 = static_cast<int64_t>(tile_m) * rows;
      if (!all_ready) {
        // no accumulators: nothing to look up
      } else if (look.stats == nullptr && spread_pays<4>(pairs, L)) {
        int* best = reinterpret_cast<int*>(sm.a[1]);
        lookup_spread<4, kCopies>(look, coordinates, best, best + pairs, pairs, tame_y, sm.inv_f, sm.lv[set], sm.primes, L, row0,
                                  tile_n * kCopies, Cg);
      } else {
        lookup_pairs<4, kCopies>(look, coordinates, pairs, tame_y, sm.inv_f, sm.lv[set], sm.primes, L, row0, tile_n * kCopies, Cg);
      }
    }
  }
  if (!ready) let_copies_land();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
  }
}

}  // namespace

bool project_tc_supported(int blocks, int ldu) { return blocks == 4 && ldu % kTileK == 0; }

void project_tc_setup(project_tc_plan& p, const __half* ut, int copies, int ldu, int sms)
{
  p.copies = copies;
  p.ldu    = ldu;
  p.sms    = sms;
  make_map(p.map_b, ut, static_cast<int64_t>(copies) * 32, ldu, kTileN);
  for (auto* f : {project_decode_tc_kernel<true, tc_mode::taps>, project_decode_tc_kernel<false, tc_mode::taps>,
                  project_decode_tc_kernel<true, tc_mode::spread>, project_decode_tc_kernel<false, tc_mode::spread>,
                  project_decode_tc_kernel<true, tc_mode::bulk>, project_decode_tc_kernel<false, tc_mode::bulk>})
    cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(sizeof(tc_smem) + 1024));
}

auto project_decode_tc(const project_tc_plan& p, const sketch_job& job, int L, const __half* shift, const float* inv_f,
                       float finest, long long* codes, __half* Yout,
                       const tc_lookup& look, int* error, cudaStream_t s) -> project_shape
{
  // |y| below this keeps |y / spacing| under the bound of the short decode at every level
  const float tame_y = finest > 0.f ? kTameLimit * finest * 0.99f : 0.f;
  if (job.m <= 0 || p.copies <= 0) return {};
  CUtensorMap b;
  std::memcpy(&b, p.map_b, sizeof(b));
  const int tiles = ((p.copies + kCopies - 1) / kCopies) * ((job.m + kTileM - 1) / kTileM);
  // rows of the caller's array are read sixteen bytes at a time where they all start on such a boundary
  const bool vec   = job.D % 4 == 0 && reinterpret_cast<uintptr_t>(job.q) % 16 == 0;
  // More tiles than the GPU has places for blocks of the spread form (half of them where two launches share it, for the
  // halves of a batch): the bulk form, a block for each of its own places. us of a search of one round, 64 copies x 128
  // dimensions, in this form and, with the line at a tile for each place of the bulk form, in the other: 1 184
  // queries (320 tiles) 104 spread and 112 bulk; halves of 800 127 bulk and 148 spread, of 1 000 134 and 173; of 1 250 164
  // bulk, 205 spread. Wider rows do not stay in the operand stages from tile to tile, and the line stays where it was:
  // 200 dimensions x 200 copies, 300 queries 101 bulk and 84 spread, but 256 x 64, 1 200 107 and 116; 512 x 64, 1 200
  // 121 and 116, 2 300 168 and 161; 960 x 48, 6 000 1 115 and 1 161.
  const int places = kBulkBlocks * p.sms, spread_places = kSpreadBlocks * p.sms / job.beside;
  const bool many  = p.ldu <= kStages * kTileK ? tiles > spread_places - sketch_blocks<1>(job) : tiles >= places;
  const auto mode  = look.table == nullptr ? tc_mode::taps : many ? tc_mode::bulk : tc_mode::spread;
  const auto pick  = [&](auto taps, auto spread, auto bulk) {
    return mode == tc_mode::taps ? taps : mode == tc_mode::spread ? spread : bulk;
  };
  const auto kernel =
    vec ? pick(project_decode_tc_kernel<true, tc_mode::taps>, project_decode_tc_kernel<true, tc_mode::spread>,
               project_decode_tc_kernel<true, tc_mode::bulk>)
        : pick(project_decode_tc_kernel<false, tc_mode::taps>, project_decode_tc_kernel<false, tc_mode::spread>,
               project_decode_tc_kernel<false, tc_mode::bulk>);
  const int sk        = mode == tc_mode::bulk ? sketch_blocks<4>(job) : sketch_blocks<1>(job);
  // Queries of a tile in the spread form: a block goes through its pairs in turns of 64, so a tile of 128 queries takes
  // four times a block's latency where three blocks of fewer would fit a multiprocessor. As few as give every place
  // a block, but not fewer than keep its threads busy in one turn. us of a search of one round, 128 a tile and these: 64
  // copies x 128 dimensions, 17 queries 48.5 and 46.0, 100 64.3 and 52.6, 300 74.8 and 62.2, 600 85.6 and 78.8, 1 000 100 and
  // 95; 8 x 64, 300 62 and 47, 1 000 66 and 53. The operands of wide rows are most of a tile's time: 256 dimensions 148
  // 68 and 58, 300 71 and 67, but 600 (48 a tile) 78.1 and 79.7, 1 000 94 and 99; 960, 999 132 and 146.
  int rows = kTileM;
  if (mode == tc_mode::spread) {
    const int tiles_n = (p.copies + kCopies - 1) / kCopies;
    const int fit     = std::max(1, (spread_places - sk) / tiles_n);
    const int least   = std::max(1, kThreads / (4 * kCopies * L));
    const int split   = std::min(kTileM, (std::max((job.m + fit - 1) / fit, least) + 3) & ~3);
    if (p.ldu <= kStages * kTileK || (p.ldu <= 2 * kStages * kTileK && split <= kTileM / 3)) rows = split;
  }
  const unsigned grid = static_cast<unsigned>(
    mode == tc_mode::bulk ? places : sk + ((p.copies + kCopies - 1) / kCopies) * ((job.m + rows - 1) / rows));
  kernel<<<grid, kThreads, sizeof(tc_smem) + 1024, s>>>(b, job, sk, rows, p.copies, L, p.ldu / kTileK, shift, inv_f, tame_y,
                                                        codes, Yout, look, error);
  const auto form = mode == tc_mode::taps ? project_form::written_out : mode == tc_mode::bulk ? project_form::bulk : project_form::spread;
  return {form, rows};
}

}  // namespace octex_b200::kernels
