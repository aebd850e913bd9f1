// Exact K nearest rows of every row of an fp16 matrix, on the tensor cores (sm_100a only): what the
// neighbor table of an index is made from (the reference calls cuVS brute force for it: hpdic/octex,
// cpp/src/neighbors/octex/detail/build_table.cuh:60-142).
//
//   t[q, r] = |x_r|^2 - 2 x_q . x_r          squared distance up to the row's own constant |x_q|^2
//
// A block takes items of one or two sets of 128 query rows and walks over all rows in tiles of 128. Per tile and
// set the 128 x 128 accumulators are one chain of tcgen05.mma (fp32 in TMEM): the fp16 rows (by TMA, 128-byte
// swizzle), then a short one whose operands are the tile's norms, each as three bf16 of eight bits, and minus a half
// for each of the three. So an accumulator is -t / 2 and the epilogue neither loads a norm nor does arithmetic: norms
// from shared memory, an FMA for each, took half of the shared memory's time (a load whose 32 lanes want the same
// 16 bytes fills the data pipe for four cycles) beside the MMAs, which read their operands from it as well. The norms
// come last: the sums before are those of the products alone and the distances against 64 bits as far off as with
// an FMA behind the MMAs (root mean square, relative, of near rows: 2.25e-7 at 96 dimensions on the unit sphere,
// 6.6e-7 at 256, 6.1e-4 at 960 non-negative ones, both ways), the neighbors found the same ones. Norms first give
// 2.2e-7, 3.3e-7 and 2.8e-4 there but 2.1e-7 instead of 1.8e-7 at 64 dimensions, and other neighbors among near ties.
// The accumulators are double buffered, so the tensor cores work on tile i + 1 while four epilogue
// warps per set read tile i (tcgen05.ld, one query row per thread) and compare with what the row has to beat. The
// query rows stay in shared memory for the whole scan when they fit (256 dimensions at most), so a tile of 128
// rows is read from the L2 cache once for 256 query rows.
//
// A row meets about K (1 + ln(n / K)) improvements in all. To start with a bar, the block first visits
// every few tiles just for the least value of each column of the tiles: where 64 of them hold a share of K, there
// are that many rows at or below, so nothing beyond is in the answer. An improvement passes three hands. The
// epilogue finds the groups of four columns that hold one (the largest accumulator of each against the bar, a
// bit), reads those again and sets them aside in shared memory, a lane its own. When one of a warp's rows has no
// room left, all are looked through and what is still wanted is noted (value, row) in one of two buffers of the
// row. A full buffer goes to a list warp, which sorts it (bitonic, a key per lane) and merges it into the row's K
// best, which stand in order in the output arrays (L2 cache), and publishes the K-th. At the end of an item all rows hand
// over at once, with nothing else left to do: then the epilogue warps merge as well, whichever row no other warp has
// taken. (Left to four list warps the end of an item took 70 us, 64 merges one after the other; us a call, so and
// now: 1 000 x 128, K = 64 438 and 272, K = 10 165 and 117, 10 007 x 64, K = 64 513 and 360, 200 001 x 128 15 100 and
// 14 700, 50 000 x 768, K = 10 4 760 and 4 650.) So the bar a row compares
// with is a buffer or two old, which costs a few more notes, and no tile waits for a merge (2 000 cycles, mostly
// the latencies of shuffles and of the L2 cache, where a tile takes 2 200).
//
// What bounds it: the MMAs. One of 128 x 128 x 16 with both operands in shared memory takes 101 cycles instead
// of 64 (128 bytes a cycle would be needed), the norms one more of them, and a tile with nothing looked at 2 200
// of the 2 700 cycles that it takes (200 001 x 128, K = 64: 11.4 of 13.8 ms; 64 dimensions 8.2 of 11.3); the rest is
// what the four warps of a set wait for one another when one of them looks through its improvements.
// 200 001 x 128, K = 64, ms: 133 with a list update per improvement; 20.5 with buffers in shared memory that the
// epilogue merges itself and norms it adds; 18.3 with list warps and norms in the MMAs; 15.0 with the groups read
// again from TMEM (instead of 64 columns kept in registers until it is known which are wanted); 14.2 with the next 32
// columns on their way while 32 are looked at, 14.5 with the norms last, 14.3 looking through without votes, 13.8 with the
// ends of the items merged by all warps. Two warps per row, a half of the columns each: 18.7.
//
// Roles: warp 0 issues the TMA copies, warps 1 and 2 the MMAs of a set (one lane issues), warp 3 makes the norm
// operands; eight epilogue warps, four per set, one per quarter of the TMEM lanes; four list warps, a quarter of the rows each.
// Every wait, on an mbarrier or a word in shared memory, is bounded; one that runs out raises a flag the other roles see, the
// block waits for its copies in flight, frees its TMEM and returns with the error word set.

#include "kernels.hpp"

#include "tc_common.cuh"

#include <algorithm>

namespace octex_b200::kernels {

namespace {

constexpr int kTile       = 128;  // query rows per set = rows per tile = TMEM lanes
constexpr int kKnnThreads = 512;  // a copy warp, an MMA warp per set, a warp for the norms, eight epilogue and four list warps
constexpr int kTmemCols   = 512;  // two accumulators of 128 fp32 columns per set
constexpr int kMaxStages  = 6;
constexpr int kNoted      = 32;   // improvements a row notes for a merge, in global memory, twice
constexpr int kHitBytes   = 640;  // of a warp's groups at one place: four values and a row per lane
constexpr uint32_t kIdleLimit = 1u << 28;  // looks of a list warp for something to merge before it gives up
constexpr int kTaken      = 1 << 9;  // of notes handed over: a warp is merging them
constexpr int kVisitsPerK = 3;    // tiles looked at for the bars, per entry of a list
constexpr uint32_t kPartBytes = kTile * kTileK * 2;  // 128 rows x 64 halves of an operand
constexpr uint32_t kNormBytes = kTile * 32;          // 128 rows x 16 bf16 of a norm operand

struct knn_ctl {
  uint64_t full[kMaxStages], empty[kMaxStages];
  uint64_t queries;
  uint64_t acc_full[2][2], acc_empty[2][2];  // [set][accumulator]
  uint64_t norms_full[2], norms_empty[2];
  uint32_t tmem_base;
  int failed;
  int place;                // of the block's notes
  int finished[8];          // items an epilogue warp is through with
  int handed[2 * kTile];    // notes of a row that are to be merged: 0, or their number, which of the two buffers, kTaken
  int have[2 * kTile];      // entries in a row's list
  float bar[2 * kTile];     // what the row's list asks for, as an accumulator
};
constexpr int kCtlBytes = 3584;
static_assert(sizeof(knn_ctl) <= kCtlBytes && kCtlBytes % 16 == 0, "control block");

/// How a block's shared memory is used.
struct knn_shape {
  int stages;    // of 64 dimensions of a tile (and of the query rows, when those do not stay)
  int resident;  // the query rows stay in shared memory
  int room;      // groups of four columns a lane may have set aside
  __host__ __device__ size_t stage_bytes() const { return (resident ? 1 : 3) * static_cast<size_t>(kPartBytes); }
  __host__ __device__ size_t query_bytes(int nkb) const { return resident ? 2 * static_cast<size_t>(nkb) * kPartBytes : 0; }
  size_t smem_bytes(int nkb) const
  {
    return 1024 + query_bytes(nkb) + stages * stage_bytes() + 3 * kNormBytes + kCtlBytes + 8 * room * kHitBytes;
  }
};

__device__ __forceinline__ void mbar_arrive(uint64_t* bar)
{
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Both TMEM instructions are warp-wide: the lanes meet first (a scan before them may have diverged).
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* r)
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

__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t (&r)[4])
{
  __syncwarp();
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
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

__device__ __forceinline__ float max3(float a, float b, float c)
{
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

/// Shared-memory descriptor of an operand of 128 rows x 16 elements, 32 bytes a row, with the 32-byte swizzle.
__device__ __forceinline__ uint64_t norm_desc(const void* tile)
{
  const uint64_t addr = (smem_u32(tile) & 0x3FFFFu) >> 4;
  return addr | (uint64_t{1} << 16) | (uint64_t{256 >> 4} << 32)  // 256 bytes between 8-row groups
         | (uint64_t{1} << 46) | (uint64_t{6} << 61);             // layout: 32-byte swizzle
}

/// The norm operand's row: three bf16 whose sum is the norm, eight bits of it each, and zeros.
__device__ __forceinline__ uint4 norm_row(float v)
{
  const unsigned h1 = __float_as_uint(v) & 0xffff0000u;
  float rest        = v - __uint_as_float(h1);
  if (!(fabsf(v) < INFINITY)) rest = 0.f;
  const unsigned h2 = __float_as_uint(rest) & 0xffff0000u;
  const unsigned h3 = __float_as_uint(rest - __uint_as_float(h2));
  return make_uint4((h1 >> 16) | h2, h3 >> 16, 0u, 0u);
}

/// A bit for each of the four values that is above the bar: the signs of bar - value, a subtraction for two of them
/// and a shift for each. (Never for NaN, nor for an infinity that equals the bar.)
__device__ __forceinline__ unsigned above_bar(const float (&v)[4], float bar)
{
  unsigned d[4];
#pragma unroll
  for (int i = 0; i < 4; i += 2)
    asm("{\n\t"
        ".reg .b64 v, b, m, r;\n\t"
        "mov.b64 v, {%2, %3};\n\t"
        "mov.b64 b, {%4, %4};\n\t"
        "mov.b64 m, {%5, %5};\n\t"
        "fma.rn.f32x2 r, v, m, b;\n\t"
        "mov.b64 {%0, %1}, r;\n\t"
        "}"
        : "=r"(d[i]), "=r"(d[i + 1])
        : "f"(v[i]), "f"(v[i + 1]), "f"(bar), "f"(-1.0f));
  return __funnelshift_l(d[0], __funnelshift_l(d[1], __funnelshift_l(d[2], d[3] >> 31, 1), 1), 1);
}

/// Sets four accumulators and the row of the first aside at the shared-memory address `at`, which moves on, where
/// `wanted` is not zero; no branch.
__device__ __forceinline__ void set_aside(unsigned wanted, uint32_t& at, uint32_t to_first, const uint32_t (&v)[4], int first)
{
  asm volatile(
    "{\n\t"
    ".reg .pred p;\n\t"
    ".reg .b32 a;\n\t"
    "setp.ne.u32 p, %1, 0;\n\t"
    "add.u32 a, %0, %2;\n\t"
    "@p st.shared.v4.b32 [%0], {%3, %4, %5, %6};\n\t"
    "@p st.shared.b32 [a], %7;\n\t"
    "@p add.u32 %0, %0, %8;\n\t"
    "}"
    : "+r"(at)
    : "r"(wanted), "r"(to_first), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(first), "n"(kHitBytes)
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

// What the rows of the blocks that are running note, a place per block. It is the module's own memory, so a call
// allocates nothing for it (in an allocation of the call: 0.7 ms): 21 MB, which the driver gives the process when it
// first launches a scan (a process that only searches has none of it) and which stay with it. A block takes a place when
// it starts and leaves it when it ends; the shared memory it needs leaves no room for a second one on its multiprocessor,
// and there are more places than multiprocessors (knn_tc looks), whatever calls run at the same time.
constexpr int kPlaces = 160;
__device__ float2 notes[static_cast<size_t>(kPlaces) * 2 * kTile * 2 * kNoted];
__device__ unsigned place_taken[kPlaces];

/// A place that no other block has, -1 when none gets free.
__device__ int take_place()
{
  unsigned sm;
  asm volatile("mov.u32 %0, %%smid;" : "=r"(sm));
  for (unsigned i = 0; i < 64u * kPlaces; i++) {
    const unsigned p = (sm + i) % kPlaces;
    if (atomicCAS(&place_taken[p], 0u, 1u) == 0u) {
      __threadfence();
      return static_cast<int>(p);
    }
  }
  return -1;
}

__device__ void leave_place(int place)
{
  if (place < 0) return;
  __threadfence();
  atomicExch(&place_taken[place], 0u);
}

template <int kRegs>
__global__ void __launch_bounds__(kKnnThreads, 1)
  knn_tc_kernel(const __grid_constant__ CUtensorMap map, const float* __restrict__ norm, int n,
                int D, int K, const knn_shape shape, int sampled, int spread, int items, int wide_items, int q_first,
                int q_count, int32_t* best_id, float* best_d, int* __restrict__ error)
{
  const int nkb = (D + kTileK - 1) / kTileK;  // steps of 64 dimensions
  extern __shared__ unsigned char raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~uintptr_t{1023});
  // [set][64 dimensions][128 x 64] query rows that stay; [stages][tile | query rows of both sets]
  __half* queries = reinterpret_cast<__half*>(base);
  __half* tiles   = reinterpret_cast<__half*>(base + shape.query_bytes(nkb));
  // norm operands of two tiles, and what multiplies them
  unsigned char* norms  = base + shape.query_bytes(nkb) + shape.stages * shape.stage_bytes();
  unsigned char* halves = norms + 2 * kNormBytes;
  knn_ctl& ctl          = *reinterpret_cast<knn_ctl*>(halves + kNormBytes);
  unsigned char* hits   = halves + kNormBytes + kCtlBytes;  // [epilogue warp][entry] of kHitBytes
  constexpr int kPart = kPartBytes / 2;     // halves

  // the same for all lanes, and known to be: what the copies and the MMAs take is then computed and kept
  // in uniform registers
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x) >> 5, 0), lane = threadIdx.x & 31;
  const int q_end  = min(q_first + q_count, n);
  const int ntiles = (n + kTile - 1) / kTile;
  const int stages = shape.stages;
  // the tiles in the order of their visits: every spread-th for the bars, then all
  const int visits = sampled + ntiles;
  auto tile_of     = [&](int visit) { return visit < sampled ? visit * spread : visit - sampled; };

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; s++) {
      mbar_init(&ctl.full[s], 1);
      mbar_init(&ctl.empty[s], 2);  // both MMA warps, also the one without a set
    }
    mbar_init(&ctl.queries, 1);
    for (int b = 0; b < 2; b++) {
      mbar_init(&ctl.norms_full[b], 1);
      mbar_init(&ctl.norms_empty[b], 2);
    }
    for (int set = 0; set < 2; set++)
      for (int b = 0; b < 2; b++) {
        mbar_init(&ctl.acc_full[set][b], 1);
        mbar_init(&ctl.acc_empty[set][b], 4);  // one arrival per epilogue warp
      }
    for (int i = 0; i < 8; i++)
      ctl.finished[i] = 0;
    for (int i = 0; i < 2 * kTile; i++)
      ctl.handed[i] = 0;
    ctl.place  = take_place();
    ctl.failed = ctl.place < 0 ? 1 : 0;
    if (ctl.place < 0) atomicExch(error, 5);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl.tmem_base)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (warp == 3) {
    // Minus a half for each of the three parts. A row's parts are in the first or the second sixteen bytes of its 32,
    // as the swizzle has it, and zeros in the others, so the halves stand in both.
    for (int i = lane; i < 2 * kTile; i += 32) {
      reinterpret_cast<uint4*>(halves)[i] = make_uint4(0xbf00bf00u, 0x0000bf00u, 0u, 0u);
      for (int b = 0; b < 2; b++)
        reinterpret_cast<uint4*>(norms + b * kNormBytes)[i] = make_uint4(0u, 0u, 0u, 0u);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem      = __shfl_sync(0xffffffffu, ctl.tmem_base, 0);
  const volatile int* stop = &ctl.failed;
  const bool placed        = ctl.place >= 0;

  // What row r of the item has handed over goes into its list, unless another warp is at it; r is the same for all
  // lanes. Which warp merges a row changes, which lane has which entry of its list does not.
  auto merge_handed = [&](int r, int q0) {
    int note = 0;
    if (lane == 0) {
      note = *static_cast<volatile int*>(&ctl.handed[r]);
      if (note != 0 && ((note & kTaken) != 0 || atomicCAS(&ctl.handed[r], note, note | kTaken) != note)) note = 0;
    }
    note = __shfl_sync(0xffffffffu, note, 0);
    if (note == 0) return;
    __threadfence_block();
    const int c = note & 255, h = *static_cast<volatile int*>(&ctl.have[r]);
    const int64_t list = static_cast<int64_t>(q0 + r - q_first) * K;
    const float last   = merge_noted<kRegs>(notes + ((static_cast<size_t>(ctl.place) * 2 * kTile + r) * 2 + (note >> 8 & 1)) * kNoted, c,
                                            h, K, best_d + list, best_id + list);
    __syncwarp();
    if (lane == 0) {
      *static_cast<volatile int*>(&ctl.have[r])  = min(K, h + c);
      *static_cast<volatile float*>(&ctl.bar[r]) = -0.5f * last;
      __threadfence_block();
      *static_cast<volatile int*>(&ctl.handed[r]) = 0;
    }
    __syncwarp();
  };

  // The block's items, 256 query rows each, the narrow ones of 128 last. Visits are counted on over them
  // (modulo 2^32, which the phases of the barriers divide).
  uint32_t v0   = 0;          // the item's first visit
  int s         = 0;          // stage ring of the copy and MMA warps
  uint32_t turn = 0;
  uint32_t q_phase = 0;
  int done_items   = 0;
  for (int item = blockIdx.x; placed && item < items; item += gridDim.x, v0 += visits, q_phase ^= 1u, done_items++) {
    const int q0   = q_first + (item + min(item, wide_items)) * kTile;
    const int sets = item < wide_items && q0 + kTile < q_end ? 2 : 1;

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
      for (int t = 0; t < visits && ok; t++) {
        for (int kb = 0; kb < nkb; kb++) {
          ok = __all_sync(0xffffffffu, mbar_wait(&ctl.empty[s], (turn & 1u) ^ 1u, stop));
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
      constexpr uint32_t idesc = (1u << 4) | (static_cast<uint32_t>(kTile >> 3) << 17) |
                                 (static_cast<uint32_t>(kTile >> 4) << 24);
      constexpr uint32_t kBothBf16  = (1u << 7) | (1u << 10);
      constexpr uint64_t kPartUnits = kPartBytes >> 4;  // of a descriptor's address
      const uint64_t stage_units    = shape.stage_bytes() >> 4;
      const uint64_t tiles_desc     = umma_desc(tiles);
      const uint64_t own_desc       = shape.resident ? umma_desc(queries + set * nkb * kPart) : tiles_desc + (1 + set) * kPartUnits;
      const bool issues = elect_one();
      const bool works  = set < sets;  // else it only passes the stages on
      bool ok           = !works || !shape.resident || __all_sync(0xffffffffu, mbar_wait(&ctl.queries, q_phase, stop));
      for (int t = 0; t < visits && ok; t++) {
        const uint32_t v = v0 + t, b = v & 1u;
        if (works) ok = __all_sync(0xffffffffu, mbar_wait(&ctl.acc_empty[set][b], ((v >> 1) & 1u) ^ 1u, stop));
        if (!ok) break;
        const uint32_t acc = tmem + (2 * b + set) * kTile;
        for (int kb = 0; kb < nkb; kb++) {
          ok = __all_sync(0xffffffffu, mbar_wait(&ctl.full[s], turn & 1u, stop));
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t db = tiles_desc + s * stage_units;
          const uint64_t da = own_desc + (shape.resident ? kb * kPartUnits : s * stage_units);
          if (!works) {
            if (lane == 0) mbar_arrive(&ctl.empty[s]);
          } else if (issues) {
#pragma unroll
            for (int k = 0; k < kTileK / 16; k++)
              if (kb * kTileK + 16 * k < D)  // beyond it a tile's columns are zero
                umma_f16(acc, da + 2 * k, db + 2 * k, idesc, kb > 0 || k > 0 ? 1u : 0u);
            umma_commit(&ctl.empty[s]);  // arrives when the MMAs reading this stage are done
          }
          __syncwarp();
          if (++s == stages) s = 0, turn++;
        }
        // the norms come last
        ok = ok && __all_sync(0xffffffffu, mbar_wait(&ctl.norms_full[b], (v >> 1) & 1u, stop));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (!works) {
          if (lane == 0) mbar_arrive(&ctl.norms_empty[b]);
        } else if (issues) {
          umma_f16(acc, norm_desc(halves), norm_desc(norms + b * kNormBytes), idesc | kBothBf16, 1u);
          umma_commit(&ctl.norms_empty[b]);
          umma_commit(&ctl.acc_full[set][b]);
        }
        __syncwarp();
      }
      if (!ok && lane == 0 && atomicExch(&ctl.failed, 1) == 0) atomicExch(error, 2);
    } else if (warp == 3) {
      // ---- norms of the rows of the tiles, as the operand of an MMA; rows beyond the matrix never win ----
      bool ok = true;
      float ahead[kTile / 32];
      auto fetch = [&](int visit) {
#pragma unroll
        for (int i = 0; i < kTile / 32; i++) {
          const int r = tile_of(visit) * kTile + i * 32 + lane;
          ahead[i]    = r < n ? __ldg(norm + r) : INFINITY;
        }
      };
      fetch(0);
      for (int t = 0; t < visits && ok; t++) {
        const uint32_t v = v0 + t, b = v & 1u;
        ok = __all_sync(0xffffffffu, mbar_wait(&ctl.norms_empty[b], ((v >> 1) & 1u) ^ 1u, stop));
        if (!ok) break;
#pragma unroll
        for (int i = 0; i < kTile / 32; i++)
          *reinterpret_cast<uint4*>(norms + b * kNormBytes + (i * 32 + lane) * 32) = norm_row(ahead[i]);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&ctl.norms_full[b]);
        if (t + 1 < visits) fetch(t + 1);
      }
      if (!ok && lane == 0 && atomicExch(&ctl.failed, 1) == 0) atomicExch(error, 4);
    } else if (const int set = (warp - 4) >> 2; set < sets) {
      // ---- epilogue: one query row per thread ----------------------------------------------------
      const int quarter  = warp & 3;  // the TMEM lanes this warp may read
      const int wrow     = q0 + set * kTile + quarter * 32;  // the warp's first query row
      const int row      = wrow + lane;
      const bool live    = row < q_end;
      float2* mine       = notes + (static_cast<size_t>(ctl.place) * 2 * kTile + set * kTile + quarter * 32 + lane) * 2 * kNoted;
      // what a row has to beat, its K-th best at the last merge, as an accumulator: t = -2 (x_q . x_r - |x_r|^2 / 2)
      float bar          = live ? -INFINITY : INFINITY;
      int count          = 0;  // improvements noted for the next merge
      int buffer         = 0;  // in which of the row's two buffers
      bool ok            = true;
      volatile int* handed      = ctl.handed + set * kTile + quarter * 32 + lane;
      volatile float* list_bar  = ctl.bar + set * kTile + quarter * 32 + lane;
      *list_bar                 = -INFINITY;
      *static_cast<volatile int*>(&ctl.have[set * kTile + quarter * 32 + lane]) = 0;
      // groups of four columns with an improvement: the four values, and the first one's row `to_first` bytes behind
      const uint32_t hit0     = smem_u32(hits) + (warp - 4) * shape.room * kHitBytes + lane * 16;
      const uint32_t to_first = 512 - 12 * lane;
      const uint32_t hit_end  = hit0 + (shape.room - 2) * kHitBytes;  // beyond it there is no room for two more
      uint32_t hit            = hit0;                               // where the next one goes
      // the notes of the rows whose lanes ask for it go to the list warps; the lanes go on in the other buffer
      auto hand_over = [&](bool asks) {
        __threadfence_block();
        for (uint32_t i = 0; __any_sync(0xffffffffu, asks && *handed != 0); i++) {
          if (i == kSpinLimit || *stop != 0) {
            ok = false;
            return;
          }
          __nanosleep(64);
        }
        if (asks) {
          *handed = buffer << 8 | count;
          buffer ^= 1;
          count = 0;
        }
        __syncwarp();
      };
      // the improvements among the groups of columns set aside; a row whose notes may not hold them hands these over first
      auto look_through = [&]() {
        const bool asks = count != 0 && count + 4 * static_cast<int>((hit - hit0) / kHitBytes) > kNoted;
        if (__any_sync(0xffffffffu, asks)) hand_over(asks);
#pragma unroll 1
        for (uint32_t e = hit0; ok && e < hit; e += kHitBytes) {
          float v[4];
          int first;
          asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                       : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
                       : "r"(e)
                       : "memory");
          asm volatile("ld.shared.b32 %0, [%1];" : "=r"(first) : "r"(e + to_first) : "memory");
#pragma unroll
          for (int i = 0; i < 4; i++)
            if (v[i] > bar && first + i != row)
              mine[buffer * kNoted + count++] = make_float2(fmaf(-2.0f, v[i], 0.0f), __int_as_float(first + i));
        }
        __syncwarp();
        hit = hit0;
      };
      // a row itself is no neighbor
      auto drop_own = [&](uint32_t* r, int first) {
        if (first < wrow + 32 && first + 32 > wrow) {
#pragma unroll
          for (int i = 0; i < 32; i++)
            if (first + i == row) r[i] = __float_as_uint(-INFINITY);
        }
      };
      // The 128 columns of an accumulator, the next 32 on their way while the ones before are looked at. The largest of
      // every four is compared with the bar, which leaves a bit for each. Of the few groups in which one of the warp's
      // rows has an improvement the columns are read once more, two groups at a time, and set aside by the rows that
      // want them: to keep them in registers for that, to choose a row's group among them by its bits or to set the
      // groups aside at once, every one under a predicate, takes longer than the second reading.
      auto scan = [&](uint32_t columns, int first) {
        auto improvements = [&](const uint32_t (&r)[32]) {
          unsigned bits = 0;
#pragma unroll
          for (int h = 0; h < 2; h++) {
            float most[4];
#pragma unroll
            for (int g = 0; g < 4; g++) {
              const uint32_t* a = r + 16 * h + 4 * g;
              most[g]           = fmaxf(max3(__uint_as_float(a[0]), __uint_as_float(a[1]), __uint_as_float(a[2])), __uint_as_float(a[3]));
            }
            bits |= above_bar(most, bar) << (4 * h);
          }
          return bits;
        };
        uint32_t r[2][32];
        unsigned own = 0;
        tmem_ld32(columns, r[0]);
#pragma unroll
        for (int c = 0; c < 4; c++) {
          tmem_ld_wait();
          if (c < 3) tmem_ld32(columns + 32 * (c + 1), r[(c + 1) & 1]);
          own |= improvements(r[c & 1]) << (8 * c);
        }
        unsigned todo = __reduce_or_sync(0xffffffffu, own);
        while (todo != 0) {
          const int g = __ffs(todo) - 1;
          todo &= todo - 1;
          const int g2 = todo != 0 ? __ffs(todo) - 1 : g;
          todo &= todo - 1;
          uint32_t v[2][4];
          tmem_ld4(columns + 4 * g, v[0]);
          tmem_ld4(columns + 4 * g2, v[1]);
          tmem_ld_wait();
          set_aside(own >> g & 1u, hit, to_first, v[0], first + 4 * g);
          set_aside(g2 != g ? own >> g2 & 1u : 0u, hit, to_first, v[1], first + 4 * g2);
          if (__any_sync(0xffffffffu, hit > hit_end)) look_through();
        }
      };
      // the accumulator of a visit is there
      auto begin = [&](int visit) {
        const uint32_t v = v0 + visit;
        ok = __all_sync(0xffffffffu, mbar_wait(&ctl.acc_full[set][v & 1u], (v >> 1) & 1u, stop));
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        return ok;
      };
      // 32 columns of the visit's accumulator; once the last are there the tensor cores may overwrite it
      const uint32_t tmem_rows = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + static_cast<uint32_t>(set * kTile);
      auto columns             = [&](int visit, int c, uint32_t* r) {
        tmem_ld32(tmem_rows + ((v0 + visit) & 1u) * 2 * kTile + static_cast<uint32_t>(c * 32), r);
      };
      auto release = [&](int visit) {
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&ctl.acc_empty[set][(v0 + visit) & 1u]);
      };
      int visit = 0;
      {
        // One largest value per column of a tile, columns 64 apart sharing one: neighbors that stand next to each
        // other in the matrix still count one by one. Longer lists take several parts of the tiles one after the
        // other and ask each for its share: where every part has K / parts rows, they have K together.
        const int parts = (K + 31) / 32, share = (K + parts - 1) / parts;
        float lowest = INFINITY;
#pragma unroll 1
        for (int part = 1; part <= parts && ok; part++) {
          float most[2][32];
#pragma unroll
          for (int c = 0; c < 2; c++)
#pragma unroll
            for (int i = 0; i < 32; i++)
              most[c][i] = -INFINITY;
          const int end = static_cast<int>(static_cast<int64_t>(sampled) * part / parts);
#pragma unroll 1
          for (; visit < end; visit++) {
            if (!begin(visit)) break;
#pragma unroll
            for (int c = 0; c < 4; c++) {
              uint32_t r[32];
              columns(visit, c, r);
              tmem_ld_wait();
              if (c == 3) release(visit);
              drop_own(r, tile_of(visit) * kTile + c * 32);
#pragma unroll
              for (int i = 0; i < 32; i++)
                most[c & 1][i] = fmaxf(most[c & 1][i], __uint_as_float(r[i]));
            }
          }
          // halving of the range between the least and the largest of them, never above `share` of them
          float low = INFINITY, high = -INFINITY;
#pragma unroll
          for (int c = 0; c < 2; c++)
#pragma unroll
            for (int i = 0; i < 32; i++) {
              low  = fminf(low, most[c][i]);
              high = fmaxf(high, most[c][i]);
            }
          auto above = [&](float value) {
            int many = 0;
#pragma unroll
            for (int c = 0; c < 2; c++)
#pragma unroll
              for (int i = 0; i < 32; i++)
                many += most[c][i] >= value ? 1 : 0;
            return many;
          };
#pragma unroll 1
          for (int step = 0; step < 12; step++) {
            const float middle = 0.5f * low + 0.5f * high;
            if (above(middle) >= share)
              low = middle;
            else
              high = middle;
          }
          lowest = fminf(lowest, fabsf(low) < 3e38f && above(low) >= share ? low : -INFINITY);
        }
        // rows as far as that may still be wanted: the bar that a row has to beat lies below it
        if (live && lowest > -INFINITY) bar = fmaf(fabsf(lowest), -2.4e-7f, lowest) - 1e-37f;
      }
#pragma unroll 1
      for (; ok && visit < visits; visit++) {
        if (!begin(visit)) break;
        bar = fmaxf(bar, *list_bar);
        scan(tmem_rows + ((v0 + visit) & 1u) * 2 * kTile, tile_of(visit) * kTile);
        release(visit);
      }
      if (ok) {
        look_through();
        hand_over(count != 0);
      }
      __threadfence_block();
      __syncwarp();
      if (lane == 0) *static_cast<volatile int*>(&ctl.finished[set * 4 + quarter]) = done_items + 1;
      // The last notes of all rows came at once: the list warps start from the first row, the others help from the last.
#pragma unroll 1
      for (int L = 31; L >= 0 && ok; L--)
        merge_handed(set * kTile + quarter * 32 + L, q0);
      for (uint32_t i = 0; ok && __any_sync(0xffffffffu, *handed != 0); i++) {
        ok = __all_sync(0xffffffffu, i < kSpinLimit && *stop == 0);
        __nanosleep(64);
      }
      if (!ok && lane == 0 && atomicExch(&ctl.failed, 1) == 0) atomicExch(error, 3);
      // the rows' own norms, four rows at a time
      __threadfence_block();
#pragma unroll 1
      for (int L0 = 0; ok && L0 < 32 && wrow + L0 < q_end; L0 += 4) {
        const int many = min(4, q_end - wrow - L0);
        int h[4];
        float qn[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
          h[u]  = u < many ? *static_cast<volatile int*>(&ctl.have[set * kTile + quarter * 32 + L0 + u]) : 0;
          qn[u] = u < many ? __ldg(norm + wrow + L0 + u) : 0.f;
        }
        float* od   = best_d + static_cast<int64_t>(wrow + L0 - q_first) * K;
        int32_t* oi = best_id + static_cast<int64_t>(wrow + L0 - q_first) * K;
        for (int t = lane; t < K; t += 32) {
          float d[4];
#pragma unroll
          for (int u = 0; u < 4; u++)
            d[u] = t < h[u] ? od[u * K + t] : INFINITY;
#pragma unroll
          for (int u = 0; u < 4; u++)
            if (u < many) {
              od[u * K + t] = t < h[u] ? fmaxf(__fadd_rn(qn[u], d[u]), 0.f) : INFINITY;
              if (t >= h[u]) oi[u * K + t] = -1;
            }
        }
      }
    } else if (warp >= 12) {
      // ---- lists: what the rows hand over is merged while the epilogue goes on; 64 rows a warp, or 32 of one set -----
      const int list = warp - 12, row0 = list * 32 * sets;  // of the block's 256
      const volatile int* handed   = ctl.handed + row0;
      const volatile int* finished = ctl.finished + list * sets;
      bool ok = true;
      for (uint32_t idle = 0; ok;) {
        const bool over = __all_sync(0xffffffffu, finished[lane & (sets - 1)] == done_items + 1);
        __threadfence_block();
        auto waits = [&](int r) {
          const int note = handed[r];
          return note != 0 && (note & kTaken) == 0;
        };
        unsigned long long todo = __ballot_sync(0xffffffffu, waits(lane));
        if (sets == 2) todo |= static_cast<unsigned long long>(__ballot_sync(0xffffffffu, waits(32 + lane))) << 32;
        if (todo == 0) {
          if (over) break;
          ok = __all_sync(0xffffffffu, *stop == 0 && ++idle < kIdleLimit);
          __nanosleep(1000);
          continue;
        }
        idle = 0;
#pragma unroll 1
        for (; todo != 0; todo &= todo - 1)
          merge_handed(row0 + __ffsll(todo) - 1, q0);
      }
      if (!ok && lane == 0 && atomicExch(&ctl.failed, 1) == 0) atomicExch(error, 6);
    }
    __syncwarp();
    // every accumulator has been read, so no MMA is left that reads the query rows
    if (__syncthreads_or(*stop)) break;
  }
  if (*stop != 0) let_copies_land();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (threadIdx.x == 0) leave_place(ctl.place);
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
  }
}

/// Query rows that stay in shared memory with as many stages as fit behind them, three at least (256 dimensions).
/// Beyond that they come in again with every tile, in four stages.
/// Four places for groups: a warp looks through them when there is no room for two more in one of its lanes, and all are
/// noted at once, so at most kNoted / 4. More hold up what the lists publish, fewer are looked through too often; us a call
/// with six, four, three and two: 200 001 x 128, K = 64 14 820, 14 560, 14 860 and 16 470, 100 000 x 128, K = 120 5 822,
/// 5 580, 5 795 and 6 725, 1 000 x 128, K = 64 272, 245, 236 and 232 (248 with lists that the epilogue merged alone). Where
/// query rows do not stay three leave the room for the fourth stage; us with four places and three stages and with three and
/// four, 50 000 rows, K = 10 and 64: 768 dimensions 4 658 and 4 516, 6 567 and 6 353, 960 5 763 and 5 508, 8 124 and 7 739,
/// 512 3 204 and 3 190, 4 488 and 4 482.
/// What these take beyond a scan whose epilogue merges alone and adds the norms itself (3 070 at 512 dimensions and K = 10,
/// 4 420 at 768; 4 610 and 6 350 at K = 64) are the MMAs of the norms; norms in the epilogue of this one 3 560 and 4 910,
/// since they come out of the shared memory the MMAs wait for. One set that stays instead of two that do not, 264 to 576
/// dimensions: 3 080 and 4 160 at 512.
knn_shape choose_shape(int nkb)
{
  constexpr size_t kLimit = 227 * 1024;
  knn_shape fit{kMaxStages, 1, 4};
  while (fit.stages > 3 && fit.smem_bytes(nkb) > kLimit)
    fit.stages--;
  return fit.smem_bytes(nkb) <= kLimit ? fit : knn_shape{4, 0, 3};
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
  if (sms > kPlaces) throw std::runtime_error("octex: more multiprocessors than the neighbor scan has places for notes");
  // A block per multiprocessor, which takes items of 256 query rows; what is left after the whole rounds goes out
  // in items of 128 rows when those fit one more round, which then takes half the time.
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
  const int64_t items  = wide + narrow;
  kernel<<<static_cast<unsigned>(std::min<int64_t>(items, sms)), kKnnThreads, smem, s>>>(
    map, norm, static_cast<int>(n), D, K, shape, static_cast<int>((ntiles + spread - 1) / spread), static_cast<int>(spread),
    static_cast<int>(items), static_cast<int>(wide), static_cast<int>(q_first), static_cast<int>(q_count), best_id, best_d,
    error);
}

}  // namespace octex_b200::kernels
