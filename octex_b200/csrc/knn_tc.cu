// Exact K nearest rows of every row of an fp16 matrix, on the tensor cores (sm_100a only): what the
// neighbor table of an index is made from (the reference calls cuVS brute force for it: hpdic/octex,
// cpp/src/neighbors/octex/detail/build_table.cuh:60-142).
//
//   t[q, r] = |x_r|^2 - 2 x_q . x_r          squared distance up to the row's own constant |x_q|^2
//
// A block owns one or two sets of 128 query rows and walks over all rows in tiles of 128. Per tile and
// set the 128 x 128 dot products are one tcgen05.mma chain (fp16 operands by TMA, 128-byte swizzle,
// fp32 accumulators in TMEM); the accumulators are double buffered, so the tensor cores work on tile
// i + 1 while four epilogue warps per set read tile i out of TMEM (tcgen05.ld, one query row per
// thread), add the row norms and compare against the worst entry the row keeps. The query rows stay in
// shared memory for the whole scan when they fit (256 dimensions at most), so a tile of 128 rows is read
// from the L2 cache once for 256 query rows.
//
// A row meets about K (1 + ln(n / K)) improvements in all. To start with a bar, the block first visits
// every few tiles just for the least value of each column of the tiles, up to 128 registers a thread: the
// K-th smallest of these has K rows at or below it, so nothing beyond it is in the answer. A thread only
// appends an improvement (value, row) to a short buffer of its row in shared memory; when one of a warp's
// rows has no room for eight more, the warp sorts that buffer (bitonic, a key per lane) and merges it into
// the row's K best, which stand in order in the output arrays (L2 cache). So the bar a row compares with is
// up to a buffer old, which costs a few more appends, and a merge of a few hundred instructions serves 16
// to 32 of them.
//
// What bounds it: the epilogue, two warps to a scheduler (168 registers a thread, and ptxas still spills 72,
// 176 and 304 bytes with one, two and four keys a lane), each at an instruction every five cycles; the
// MMAs are 29 % of a tile's time (262 144 x 128, K = 64: 30.2 ms, tensor pipe 28.9 %, issue slots 40.7 % busy).
// 200 001 x 128, K = 64: 133 ms with a list update per improvement and a list per half of the tiles; 26 with
// buffers and resident query rows; 21 with the bars, a warp per set for the MMAs, operands in uniform
// registers, and one mask of the groups of columns that hold improvements where there was a vote and a
// branch for each.
//
// Roles: warp 0 issues the TMA copies, warps 1 and 2 the MMAs of a set (one lane issues); the other warps
// are the epilogue, in sets of four (one per quarter of the TMEM lanes).
// Every wait on an mbarrier is bounded; a wait that runs out raises a flag the other roles see, the
// block waits for its copies in flight, frees its TMEM and returns with the error word set.

#include "kernels.hpp"

#include "tc_common.cuh"

#include <algorithm>

namespace octex_b200::kernels {

namespace {

constexpr int kTile       = 128;  // query rows per set = rows per tile = TMEM lanes
constexpr int kKnnThreads = 352;  // copy warp, an MMA warp per set, two sets of four epilogue warps
constexpr int kTmemCols   = 512;  // two accumulators of 128 fp32 columns per set
constexpr int kMaxStages  = 6;
constexpr int kVisitsPerK = 3;    // tiles looked at for the bars, per entry of a list
constexpr uint32_t kPartBytes = kTile * kTileK * 2;  // 128 rows x 64 halves of an operand

struct knn_ctl {
  uint64_t full[kMaxStages], empty[kMaxStages];
  uint64_t queries;
  uint64_t acc_full[2][2], acc_empty[2][2];  // [set][accumulator]
  uint32_t tmem_base;
  int failed;
  alignas(16) float nb[8][kTile];  // norms of the rows of the tile an epilogue warp works on
};
constexpr int kCtlBytes = 4608;
static_assert(sizeof(knn_ctl) <= kCtlBytes && kCtlBytes % 16 == 0, "control block");

/// How a block's shared memory is used.
struct knn_shape {
  int stages;    // of 64 dimensions of a tile (and of the query rows, when those do not stay)
  int room;      // noted improvements per row: 32 or 16
  int resident;  // the query rows stay in shared memory
  __host__ __device__ size_t stage_bytes() const { return (resident ? 1 : 3) * static_cast<size_t>(kPartBytes); }
  __host__ __device__ size_t query_bytes(int nkb) const { return resident ? 2 * static_cast<size_t>(nkb) * kPartBytes : 0; }
  size_t smem_bytes(int nkb) const
  {
    return 1024 + query_bytes(nkb) + stages * stage_bytes() + kCtlBytes + 2 * kTile * static_cast<size_t>(room + 1) * 8;
  }
};

__device__ __forceinline__ void mbar_arrive(uint64_t* bar)
{
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Both TMEM instructions are warp-wide: the lanes meet first (a scan before them may have diverged).
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32])
{
  __syncwarp();
  asm volatile(
    "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
    "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
    "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
      "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
      "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]),
      "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]),
      "=r"(r[30]), "=r"(r[31])
    : "r"(taddr)
    : "memory");
}

__device__ __forceinline__ void tmem_ld_wait()
{
  __syncwarp();
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

/// True in one lane of the warp, always the same.
__device__ __forceinline__ bool elect_one()
{
  uint32_t p;
  asm volatile(
    "{\n\t"
    ".reg .pred p;\n\t"
    "elect.sync _|p, 0xffffffff;\n\t"
    "selp.u32 %0, 1, 0, p;\n\t"
    "}"
    : "=r"(p));
  return p != 0;
}

/// (a, b) * -2 + (x, y): two fused multiply-adds in one instruction.
__device__ __forceinline__ void minus_twice(uint32_t a, uint32_t b, float x, float y, float& u, float& v)
{
  asm("{\n\t"
      ".reg .b64 ab, xy, m2, r;\n\t"
      "mov.b64 ab, {%2, %3};\n\t"
      "mov.b64 xy, {%4, %5};\n\t"
      "mov.b64 m2, {%6, %6};\n\t"
      "fma.rn.f32x2 r, ab, m2, xy;\n\t"
      "mov.b64 {%0, %1}, r;\n\t"
      "}"
      : "=f"(u), "=f"(v)
      : "r"(a), "r"(b), "f"(x), "f"(y), "f"(-2.0f));
}

__device__ __forceinline__ float min3(float a, float b, float c)
{
  float d;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

/// Appends (value, row) at the shared-memory address `at` when the value is below the bar; no branch.
__device__ __forceinline__ void note_below(float value, float bar, int row, uint32_t& at)
{
  asm volatile(
    "{\n\t"
    ".reg .pred p;\n\t"
    "setp.lt.f32 p, %1, %2;\n\t"
    "@p st.shared.b32 [%0], %1;\n\t"
    "@p st.shared.b32 [%0 + 4], %3;\n\t"
    "@p add.u32 %0, %0, 8;\n\t"
    "}"
    : "+r"(at)
    : "f"(value), "f"(bar), "r"(row)
    : "memory");
}

/// Keys in the order of (value, row); no value is NaN or -0.
__device__ __forceinline__ unsigned long long order_key(float v, int32_t id)
{
  const unsigned u = __float_as_uint(v);
  return (static_cast<unsigned long long>(u ^ ((u & 0x80000000u) ? 0xffffffffu : 0x80000000u)) << 32) |
         static_cast<unsigned>(id);
}
__device__ __forceinline__ float key_value(unsigned long long k)
{
  const unsigned u = static_cast<unsigned>(k >> 32);
  return __uint_as_float(u ^ ((u & 0x80000000u) ? 0x80000000u : 0xffffffffu));
}

/// A step of a bitonic network between lanes `stride` apart; the lower lane takes the smaller key when up.
__device__ __forceinline__ unsigned long long exchange(unsigned long long k, int stride, bool up)
{
  const unsigned long long other = __shfl_xor_sync(0xffffffffu, k, stride);
  const bool smaller             = ((threadIdx.x & stride) == 0) == up;
  return (k < other) == smaller ? k : other;
}

/// The warp's merge of `count` <= 32 noted entries into a row's list: `have` entries in order in
/// vals / ids (slot i * 32 + lane belongs to the lane, so no ordering between lanes is needed in memory).
/// Returns the K-th value, +inf while there are fewer. kRegs * 32 >= K.
template <int kRegs>
__device__ __forceinline__ float merge_noted(const float2* noted, int count, int have, int K, float* vals, int32_t* ids)
{
  const int lane = threadIdx.x & 31;
  unsigned long long key[kRegs];
#pragma unroll
  for (int i = 0; i < kRegs; i++) {
    const int at = i * 32 + lane;
    key[i]       = ~0ULL;
    if (at < have) key[i] = order_key(vals[at], ids[at]);
  }
  unsigned long long add = ~0ULL;
  if (lane < count) {
    const float2 e = noted[lane];
    add            = order_key(e.x, __float_as_int(e.y));
  }
  // descending, so that lane j meets the list's entry j of the last 32: of two sorted sequences the
  // smaller ones of opposite pairs are the smallest and form a bitonic sequence
#pragma unroll
  for (int size = 2; size <= 32; size <<= 1)
#pragma unroll
    for (int stride = size >> 1; stride > 0; stride >>= 1)
      add = exchange(add, stride, size < 32 && (lane & size) != 0);
  key[kRegs - 1] = min(key[kRegs - 1], add);
#pragma unroll
  for (int half = kRegs / 2; half > 0; half >>= 1)
#pragma unroll
    for (int i = 0; i < kRegs; i++)
      if ((i & half) == 0) {
        const unsigned long long a = key[i], b = key[i + half];
        key[i]        = min(a, b);
        key[i + half] = max(a, b);
      }
#pragma unroll
  for (int i = 0; i < kRegs; i++)
#pragma unroll
    for (int stride = 16; stride > 0; stride >>= 1)
      key[i] = exchange(key[i], stride, true);
  const int now = min(K, have + count);
  float last    = INFINITY;
#pragma unroll
  for (int i = 0; i < kRegs; i++) {
    const int at  = i * 32 + lane;
    const float v = key_value(key[i]);
    if (at < now) {
      vals[at] = v;
      ids[at]  = static_cast<int32_t>(key[i] & 0xffffffffu);
    }
    const float kth = __shfl_sync(0xffffffffu, v, (K - 1) & 31);
    if (i == (K - 1) >> 5 && now == K) last = kth;
  }
  return last;
}

template <int kRegs>
__global__ void __launch_bounds__(kKnnThreads, 1)
  knn_tc_kernel(const __grid_constant__ CUtensorMap map, const float* __restrict__ norm, int n,
                int D, int K, const knn_shape shape, int sampled, int spread, int wide_blocks, int q_first, int q_count,
                int32_t* best_id, float* best_d, int* __restrict__ error)
{
  const int nkb = (D + kTileK - 1) / kTileK;  // steps of 64 dimensions
  extern __shared__ unsigned char raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~uintptr_t{1023});
  // [set][64 dimensions][128 x 64] query rows that stay; [stages][tile | query rows of both sets]
  __half* queries = reinterpret_cast<__half*>(base);
  __half* tiles   = reinterpret_cast<__half*>(base + shape.query_bytes(nkb));
  unsigned char* after = base + shape.query_bytes(nkb) + shape.stages * shape.stage_bytes();
  knn_ctl& ctl    = *reinterpret_cast<knn_ctl*>(after);
  float2* noted   = reinterpret_cast<float2*>(after + kCtlBytes);  // [set][row][room + 1]
  constexpr int kPart = kPartBytes / 2;                            // halves

  // the same for all lanes, and known to be: what the copies and the MMAs take is then computed and kept
  // in uniform registers
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x) >> 5, 0), lane = threadIdx.x & 31;
  const bool wide  = static_cast<int>(blockIdx.x) < wide_blocks;
  const int q_end  = min(q_first + q_count, n);
  const int q0     = q_first + (static_cast<int>(blockIdx.x) + min(static_cast<int>(blockIdx.x), wide_blocks)) * kTile;
  const int sets   = wide && q0 + kTile < q_end ? 2 : 1;
  const int ntiles = (n + kTile - 1) / kTile;
  const int stages = shape.stages;
  // the tiles in the order of their visits: every spread-th for the bars, then all
  const int visits = sampled + ntiles;
  auto tile_of     = [&](int visit) { return visit < sampled ? visit * spread : visit - sampled; };

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; s++) {
      mbar_init(&ctl.full[s], 1);
      mbar_init(&ctl.empty[s], sets);
    }
    mbar_init(&ctl.queries, 1);
    for (int set = 0; set < 2; set++)
      for (int b = 0; b < 2; b++) {
        mbar_init(&ctl.acc_full[set][b], 1);
        mbar_init(&ctl.acc_empty[set][b], 4);  // one arrival per epilogue warp
      }
    ctl.failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl.tmem_base)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem      = __shfl_sync(0xffffffffu, ctl.tmem_base, 0);
  const volatile int* stop = &ctl.failed;

  if (warp == 0) {
    // ---- copies: the warp goes through the loop together, one lane issues --------------------------
    const bool issues = elect_one();
    bool ok           = true;
    if (shape.resident && issues) {
      mbar_expect_tx(&ctl.queries, static_cast<uint32_t>(sets * nkb) * kPartBytes);
      for (int set = 0; set < sets; set++)
        for (int kb = 0; kb < nkb; kb++)
          tma_load_2d(queries + (set * nkb + kb) * kPart, &map, kb * kTileK, q0 + set * kTile, &ctl.queries);
    }
    int s         = 0;
    uint32_t turn = 0;
    for (int t = 0; t < visits && ok; t++) {
      for (int kb = 0; kb < nkb; kb++) {
        if (turn > 0) ok = __all_sync(0xffffffffu, mbar_wait(&ctl.empty[s], (turn & 1u) ^ 1u, stop));
        if (!ok) break;
        __half* b = tiles + s * (shape.stage_bytes() / 2);
        if (issues) {
          mbar_expect_tx(&ctl.full[s], shape.resident ? kPartBytes : kPartBytes * (1 + sets));
          tma_load_2d(b, &map, kb * kTileK, tile_of(t) * kTile, &ctl.full[s]);
          if (!shape.resident)
            for (int set = 0; set < sets; set++)
              tma_load_2d(b + (1 + set) * kPart, &map, kb * kTileK, q0 + set * kTile, &ctl.full[s]);
        }
        __syncwarp();
        if (++s == stages) s = 0, turn++;
      }
    }
    if (!ok && lane == 0 && atomicExch(&ctl.failed, 1) == 0) atomicExch(error, 1);
  } else if (warp <= 2) {
    // ---- MMAs: a warp per set, so that one set's waits pass under the other's MMAs ----------------
    const int set = warp - 1;
    if (set < sets) {
      constexpr uint32_t idesc = (1u << 4) | (static_cast<uint32_t>(kTile >> 3) << 17) |
                                 (static_cast<uint32_t>(kTile >> 4) << 24);
      constexpr uint64_t kPartUnits = kPartBytes >> 4;  // of a descriptor's address
      const uint64_t stage_units    = shape.stage_bytes() >> 4;
      const uint64_t tiles_desc     = umma_desc(tiles);
      const uint64_t own_desc       = shape.resident ? umma_desc(queries + set * nkb * kPart) : tiles_desc + (1 + set) * kPartUnits;
      const bool issues = elect_one();
      bool ok           = !shape.resident || __all_sync(0xffffffffu, mbar_wait(&ctl.queries, 0, stop));
      int s             = 0;
      uint32_t turn     = 0;
      for (int t = 0; t < visits && ok; t++) {
        const int b      = t & 1;
        const uint32_t u = static_cast<uint32_t>(t >> 1);
        if (t >= 2) ok = __all_sync(0xffffffffu, mbar_wait(&ctl.acc_empty[set][b], (u & 1u) ^ 1u, stop));
        if (!ok) break;
        const uint32_t acc = tmem + static_cast<uint32_t>((2 * b + set) * kTile);
        for (int kb = 0; kb < nkb; kb++) {
          ok = __all_sync(0xffffffffu, mbar_wait(&ctl.full[s], turn & 1u, stop));
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t db = tiles_desc + s * stage_units;
          const uint64_t da = own_desc + (shape.resident ? kb * kPartUnits : s * stage_units);
          if (issues) {
#pragma unroll
            for (int k = 0; k < kTileK / 16; k++)
              if (kb * kTileK + 16 * k < D)  // beyond it a tile's columns are zero
                umma_f16(acc, da + 2 * k, db + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
            umma_commit(&ctl.empty[s]);  // arrives when the MMAs reading this stage are done
            if (kb + 1 == nkb) umma_commit(&ctl.acc_full[set][b]);
          }
          __syncwarp();
          if (++s == stages) s = 0, turn++;
        }
      }
      if (!ok && lane == 0 && atomicExch(&ctl.failed, 1) == 0) atomicExch(error, 2);
    }
  } else if (const int set = (warp - 3) >> 2; set < sets) {
    // ---- epilogue: one query row per thread ----------------------------------------------------
    const int quarter  = warp & 3;  // the TMEM lanes this warp may read
    const int wrow     = q0 + set * kTile + quarter * 32;  // the warp's first query row
    const int row      = wrow + lane;
    const bool live    = row < q_end;
    const int room     = shape.room;
    float2* rows_noted = noted + static_cast<size_t>(set * kTile + quarter * 32) * (room + 1);  // of the warp's 32 rows
    float2* mine       = rows_noted + lane * (room + 1);  // an odd number of entries apart: no bank conflicts either way
    int32_t* ids       = best_id + static_cast<int64_t>(wrow - q_first) * K;
    float* vals        = best_d + static_cast<int64_t>(wrow - q_first) * K;
    float kth          = live ? INFINITY : -INFINITY;  // what a row has to beat: its K-th best at the last merge
    int have           = 0;                            // entries of the row in the output arrays
    const uint32_t at0     = smem_u32(mine);
    const uint32_t last_at = at0 + 8 * (room - 8);  // beyond it there is no room for eight more
    uint32_t at            = at0;                   // where the next improvement goes
    float* nb              = ctl.nb[warp - 3];
    auto merge_rows = [&](unsigned which) {
      while (which != 0) {
        const int L = __ffs(which) - 1;
        which &= which - 1;
        const int c = static_cast<int>(__shfl_sync(0xffffffffu, at - at0, L) >> 3), h = __shfl_sync(0xffffffffu, have, L);
        __syncwarp();
        const float last = merge_noted<kRegs>(rows_noted + L * (room + 1), c, h, K, vals + static_cast<int64_t>(L) * K,
                                              ids + static_cast<int64_t>(L) * K);
        __syncwarp();
        if (lane == L) {
          kth  = fminf(kth, last);
          have = min(K, h + c);
          at   = at0;
        }
      }
    };
    // t of 32 columns; a row itself is infinitely far
    auto distances = [&](const uint32_t (&r)[32], int col, int first, float* d) {
#pragma unroll
      for (int g = 0; g < 8; g++) {
        const float4 nn = *reinterpret_cast<const float4*>(nb + col + g * 4);
        minus_twice(r[g * 4 + 0], r[g * 4 + 1], nn.x, nn.y, d[g * 4 + 0], d[g * 4 + 1]);
        minus_twice(r[g * 4 + 2], r[g * 4 + 3], nn.z, nn.w, d[g * 4 + 2], d[g * 4 + 3]);
      }
      if (first < wrow + 32 && first + 32 > wrow) {
#pragma unroll
        for (int i = 0; i < 32; i++)
          if (first + i == row) d[i] = INFINITY;
      }
    };
    // 64 columns of the tile: the least of every eight is looked at first; where one of the warp's rows
    // has an improvement among them, every thread appends its own; a row without room for eight more is
    // merged. (A vote and a branch per eight columns: 25 ms where this takes 21.)
    auto scan = [&](const uint32_t (&r)[2][32], int col, int first) {
      float d[64];
      distances(r[0], col, first, d);
      distances(r[1], col + 32, first + 32, d + 32);
      float least[8];
#pragma unroll
      for (int g = 0; g < 8; g++)
        least[g] = fminf(min3(min3(d[8 * g], d[8 * g + 1], d[8 * g + 2]), d[8 * g + 3], d[8 * g + 4]),
                         min3(d[8 * g + 5], d[8 * g + 6], d[8 * g + 7]));
      const float all = fminf(min3(min3(least[0], least[1], least[2]), least[3], least[4]), min3(least[5], least[6], least[7]));
      if (!__any_sync(0xffffffffu, all < kth)) return;
      // groups of eight with an improvement, of the thread and of the warp
      unsigned own = 0;
#pragma unroll
      for (int g = 0; g < 8; g++)
        own |= least[g] < kth ? 1u << g : 0u;
      unsigned todo = __reduce_or_sync(0xffffffffu, own);
      while (todo != 0) {
        // all of them at once when every row has the room, else one by one
        const bool room_for_all = __all_sync(0xffffffffu, at + 64 * __popc(own & todo) <= last_at + 64);
        const unsigned now      = room_for_all ? todo : todo & (0u - todo);
#pragma unroll
        for (int g = 0; g < 8; g++)
          if (now & (1u << g)) {
#pragma unroll
            for (int i = 0; i < 8; i++)
              note_below(d[8 * g + i], kth, first + 8 * g + i, at);
          }
        todo ^= now;
        const unsigned full = __ballot_sync(0xffffffffu, at > last_at);
        if (full != 0) merge_rows(full);
      }
    };
    // norms of the rows of a visit's tile, four per lane; rows beyond the matrix never win
    auto fetch_norms = [&](int visit, float (&v)[4]) {
      const int first = tile_of(visit) * kTile + lane;
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int r = first + i * 32;
        v[i]        = r < n ? __ldg(norm + r) : INFINITY;
      }
    };
    float ahead[4];
    fetch_norms(0, ahead);
    bool ok = true;
    // the accumulator of a visit is there, and so are the norms of its tile
    auto begin = [&](int visit) {
      __syncwarp();  // every lane is done with the norms of the tile before
#pragma unroll
      for (int i = 0; i < 4; i++)
        nb[i * 32 + lane] = ahead[i];
      fetch_norms(visit + 1, ahead);  // in flight behind this tile
      __syncwarp();
      ok = __all_sync(0xffffffffu, mbar_wait(&ctl.acc_full[set][visit & 1], static_cast<uint32_t>(visit >> 1) & 1u, stop));
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      return ok;
    };
    // 32 columns of the visit's accumulator; once the last are there the tensor cores may overwrite it
    const uint32_t tmem_rows = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + static_cast<uint32_t>(set * kTile);
    auto columns             = [&](int visit, int c, uint32_t (&r)[32]) {
      tmem_ld32(tmem_rows + static_cast<uint32_t>(visit & 1) * 2 * kTile + static_cast<uint32_t>(c * 32), r);
    };
    auto arrived = [&](int visit, bool last) {
      tmem_ld_wait();
      if (last) {
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&ctl.acc_empty[set][visit & 1]);
      }
    };
    int visit = 0;
    {
      // one least value per column of a tile, columns 32 kParts apart sharing one: neighbors that stand
      // next to each other in the matrix still count one by one
      constexpr int kParts = kRegs == 1 ? 2 : kRegs == 2 ? 3 : 4;
      float least[kParts][32];
#pragma unroll
      for (int c = 0; c < kParts; c++)
#pragma unroll
        for (int i = 0; i < 32; i++)
          least[c][i] = INFINITY;
#pragma unroll 1
      for (; visit < sampled; visit++) {
        if (!begin(visit)) break;
#pragma unroll
        for (int c = 0; c < 4; c++) {
          uint32_t r[32];
          float d[32];
          columns(visit, c, r);
          arrived(visit, c == 3);
          distances(r, c * 32, tile_of(visit) * kTile + c * 32, d);
#pragma unroll
          for (int i = 0; i < 32; i++)
            least[c % kParts][i] = fminf(least[c % kParts][i], d[i]);
        }
      }
      // halving of the range between the least and the largest of them, never below K of them
      float low = INFINITY, high = -INFINITY;
#pragma unroll
      for (int c = 0; c < kParts; c++)
#pragma unroll
        for (int i = 0; i < 32; i++) {
          low  = fminf(low, least[c][i]);
          high = fmaxf(high, least[c][i]);
        }
      auto below = [&](float bar) {
        int many = 0;
#pragma unroll
        for (int c = 0; c < kParts; c++)
#pragma unroll
          for (int i = 0; i < 32; i++)
            many += least[c][i] <= bar ? 1 : 0;
        return many;
      };
#pragma unroll 1
      for (int step = 0; step < 12; step++) {
        const float middle = 0.5f * low + 0.5f * high;
        if (below(middle) >= K)
          high = middle;
        else
          low = middle;
      }
      // rows as far as the bar may still be wanted: the bar that a row has to beat lies above it
      if (live && fabsf(high) < 3e38f && below(high) >= K) kth = fmaf(fabsf(high), 2.4e-7f, high) + 1e-37f;
    }
#pragma unroll 1
    for (; ok && visit < visits; visit++) {
      if (!begin(visit)) break;
#pragma unroll 1
      for (int c = 0; c < 4; c += 2) {
        uint32_t r[2][32];
        columns(visit, c, r[0]);
        columns(visit, c + 1, r[1]);
        arrived(visit, c == 2);
        scan(r, c * 32, tile_of(visit) * kTile + c * 32);
      }
    }
    if (!ok && lane == 0 && atomicExch(&ctl.failed, 1) == 0) atomicExch(error, 3);
    if (ok) {
      merge_rows(__ballot_sync(0xffffffffu, at != at0));
      for (int L = 0; L < 32 && wrow + L < q_end; L++) {
        const int h    = __shfl_sync(0xffffffffu, have, L);
        const float qn = __ldg(norm + wrow + L);
        float* od      = vals + static_cast<int64_t>(L) * K;
        for (int t = lane; t < K; t += 32) {
          od[t] = t < h ? fmaxf(__fadd_rn(qn, od[t]), 0.f) : INFINITY;
          if (t >= h) ids[static_cast<int64_t>(L) * K + t] = -1;
        }
      }
    }
  }
  __syncwarp();
  if (*stop != 0) let_copies_land();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
  }
}

/// Query rows that stay in shared memory with as many stages as fit behind them; buffers of half the
/// length buy the third stage at 256 dimensions. Beyond that they come in again with every tile.
knn_shape choose_shape(int nkb)
{
  constexpr size_t kLimit = 227 * 1024;
  for (const knn_shape s : {knn_shape{kMaxStages, 32, 1}, knn_shape{kMaxStages, 16, 1}}) {
    knn_shape fit = s;
    while (fit.stages > 3 && fit.smem_bytes(nkb) > kLimit)
      fit.stages--;
    if (fit.smem_bytes(nkb) <= kLimit) return fit;
  }
  return knn_shape{3, 32, 0};
}

}  // namespace

bool knn_tc_supported(int64_t n, int D, int K)
{
  // rows must start on 16-byte boundaries for the tensor map; ids are 32-bit
  return D % 8 == 0 && K >= 1 && K <= 122 && n < (int64_t{1} << 31) - 2 * kTile;
}

void knn_tc(const __half* x, const float* norm, int64_t n, int D, int K, int64_t q_first, int64_t q_count,
            int32_t* best_id, float* best_d, int* error, cudaStream_t s)
{
  if (q_count <= 0 || n <= 0) return;
  if (!knn_tc_supported(n, D, K)) throw std::runtime_error("octex: shape not covered by the tensor-core neighbor scan");
  CUtensorMap map;
  make_map(&map, x, n, D, kTile);
  const int nkb         = (D + kTileK - 1) / kTileK;
  const knn_shape shape = choose_shape(nkb);
  const size_t smem     = shape.smem_bytes(nkb);
  const auto kernel     = K <= 32 ? knn_tc_kernel<1> : K <= 64 ? knn_tc_kernel<2> : knn_tc_kernel<4>;
  cudaError_t status    = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxBlockSmem);
  int dev = 0, sms = 1;
  if (status == cudaSuccess) status = cudaGetDevice(&dev);
  if (status == cudaSuccess) status = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (status != cudaSuccess) throw std::runtime_error(std::string("octex: ") + cudaGetErrorString(status));
  // A block per multiprocessor, 256 query rows each; what is left after the whole rounds goes out in
  // blocks of 128 rows when those fit one more round, which then takes half the time.
  const int64_t round  = int64_t{2} * kTile * sms;
  const int64_t rest   = q_count % round;
  const int64_t narrow = rest <= round / 2 ? (rest + kTile - 1) / kTile : 0;
  // Tiles that are looked at for the bars: a visit costs the same whatever it saves, an improvement the
  // same work at any n, and K ln(n / visits) of them are left: the best number of visits grows with K
  // alone. 266 665 x 96, K = 64: 34.5 ms with 16 visits, 33.5 with 2 K and 4 K, 45.5 with every tile.
  // With fewer tiles than that (24 576 rows at K = 64) all of them are looked at, which still pays: 3 000 x
  // 128, K = 64, 0.95 ms a call and 1.16 without the bars, 16 000 1.29 and 1.63, K = 100 1.58 and 2.22.
  const int64_t ntiles = (n + kTile - 1) / kTile;
  const int64_t spread = std::max<int64_t>(1, ntiles / std::max(16, kVisitsPerK * K));
  const int64_t wide   = narrow > 0 || rest == 0 ? (q_count - rest) / (2 * kTile) : (q_count + 2 * kTile - 1) / (2 * kTile);
  kernel<<<static_cast<unsigned>(wide + narrow), kKnnThreads, smem, s>>>(
    map, norm, static_cast<int>(n), D, K, shape, static_cast<int>((ntiles + spread - 1) / spread), static_cast<int>(spread),
    static_cast<int>(wide), static_cast<int>(q_first), static_cast<int>(q_count), best_id, best_d, error);
}

}  // namespace octex_b200::kernels
