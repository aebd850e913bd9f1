// One round of the search per query block (sm_100a): gather, dedup, sketch scoring, selection,
// exact rerank and merge into the kept list in one kernel; for waves the choice of the start points
// comes first in the same kernel. A query's candidates stay in shared memory from the first list
// entry to the kept list.
//
// Semantics follow the reference's per-step kernels (hpdic/octex,
// cpp/src/neighbors/octex/detail/search_kernels.cuh): gather_kernel :138-253, select_smallest
// :259-322, exact_distances :325-342, load_keys / bitonic_sort / store_keys :345-415,
// rerank_keep_kernel :421-467, sketch_keep_kernel :471-508, merge_kept_kernel :517-564,
// pick_starts_kernel :571-631, final_rerank_kernel :634-669. What differs is how the work is laid
// out: the kept list is never fully re-sorted (the best KO keys are selected by radix passes and
// only those are sorted), candidates already in the kept list are not reranked again (their key is
// already there), and every thread keeps several independent loads in flight.

#include "kernels.hpp"

#include "prep_common.cuh"

#include <algorithm>
#include <cfloat>
#include <cmath>

namespace octex_b200::kernels {

namespace {

constexpr unsigned kIdHash          = 2654435761u;
constexpr unsigned long long kNoKey = ~0ULL;
constexpr int kAheadBytes           = 512;  // fp16 rows up to this are asked for ahead of the exact distances

/// Words every thread of a block shares: counters, and what a selection finds out.
enum ctl {
  kEmitted,   // keys taken by a selection
  kBin,       // bin of the R-th key, keys still needed from it, its size
  kLeft,
  kSize,
  kDistinct,  // distinct ids of the gather
  kStarts,    // start points of a wave
  kMerged,    // new keys of a merge
  kSide,      // members of the bin of the R-th key
  kLow,       // range of the high words a selection bins
  kHigh,
  kValid,     // entries of the kept list with an id
  kWithin,    // ranking by sketch distance: candidates below the last key of a full kept list
  kCtlWords
};

/// Offsets (in 4-byte words) of the regions of a round block's shared memory.
struct round_layout {
  int table, cand, dist, pool, sorted, sid, sdv, qv, sc, fq, st, len, hist, wsum, ctrl, kid, kd, words;
  __host__ __device__ explicit round_layout(const round_args& a)
  {
    const int in_smem = a.cand_global == nullptr ? a.nmax : 0;
    const int rm      = a.sketch_rank ? a.KO : a.R;
    int at            = 0;
    auto take         = [&](int n) {
      int o = at;
      at += (n + 3) & ~3;  // keep every region 16-byte aligned
      return o;
    };
    // Two regions are used twice. The sketch distances are written where the hash set of the gather
    // was (the set is dead once the ids are collected), and the small set of kept ids is built there after
    // them (once the selection has copied out the distances it took). The keys of the merge are written where
    // the candidates were (dead after the selection).
    const int pool_words = 2 * (a.KO + rm);
    const int sort_words = a.P > 32 ? 4 * a.P : 128;  // 2 P keys, 64 at least (the one-warp sort)
    table  = take(a.ht_slots > in_smem ? a.ht_slots : in_smem);
    dist   = table;
    cand   = take(in_smem > pool_words + sort_words ? in_smem : pool_words + sort_words);
    pool   = cand;
    sorted = cand + pool_words;
    sid    = take(rm);
    sdv    = take(rm);
    // first round: 16-bit weights of the integer sketch distance (two per word) and its per-query
    // constants (-2 alpha, sum of q^2); waves: the sketch-space query and the scales as floats
    qv     = take(a.sw);
    sc     = take(a.sw);
    fq     = take((a.D + 63) & ~63);  // in 64-element steps (query_slot)
    st     = take(a.nseg);
    len    = take(a.nseg);
    hist   = take(256);
    wsum   = take(32);  // one word per warp
    ctrl   = take(kCtlWords);
    kid    = take(a.KO);
    kd     = take(a.KO);
    words  = at;
  }
};

/// Home slot of an id in a set of `slots` (any size): the high word of hash * slots.
__device__ __forceinline__ unsigned home_slot(int id, int slots)
{
  return __umulhi(static_cast<unsigned>(id) * kIdHash, static_cast<unsigned>(slots));
}

/// Exclusive prefix of v over the block (kThreads threads); total = the sum. wsum: kThreads / 32 words that
/// nothing else uses until the block's next barrier.
template <int kThreads = kRoundThreads>
__device__ __forceinline__ int block_scan(int v, int* wsum, int& total)
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int inc        = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += u;
  }
  if (lane == 31) wsum[warp] = inc;
  __syncthreads();
  const int w = lane < kThreads / 32 ? wsum[lane] : 0;
  total       = __reduce_add_sync(0xffffffffu, w);
  return __reduce_add_sync(0xffffffffu, lane < warp ? w : 0) + inc - v;
}

/// True when an id was not in the set of the gather yet and is now. The steps grow by one slot each (the
/// longest way among the 32 ids of a warp is what a step of the gather takes, and ways grow together into
/// runs where every step is one slot); from kGrowing steps on, one slot each, so that a free slot is met.
/// There is one: as many slots as entries. Against steps of one slot, thousand cycles of a block's gathers:
/// 16 384 entries and 21 848 slots, three waves, 115 and 105; 32 768 in as many slots 171 and 121 (the search
/// 4 888 and 4 340 us). Reading a slot before the exchange, or four entries' exchanges side by side, take
/// longer (179 and 178 for the first): what counts is how many steps a warp makes, and the reads come on top.
__device__ __forceinline__ bool claim(int* set, int slots, int id)
{
  constexpr int kGrowing = 32;
  unsigned s             = home_slot(id, slots);
#pragma unroll 1
  for (int p = 1; p < kGrowing + slots; p++) {
    const int was = atomicCAS(&set[s], -1, id);
    if (was == -1) return true;
    if (was == id) return false;
    s += p < kGrowing ? p : 1;
    if (s >= static_cast<unsigned>(slots)) s -= slots;
  }
  return false;
}

/// Puts an id (none when negative) into a small set of `slots` (a power of two, never full) ids.
__device__ __forceinline__ void insert_id(int* set, int slots, int id)
{
  if (id < 0) return;
  unsigned h = (static_cast<unsigned>(id) * kIdHash) & (slots - 1);
  for (int p = 0; p < slots; p++) {
    const int prev = atomicCAS(&set[h], -1, id);
    if (prev == -1 || prev == id) return;
    h = (h + 1) & (slots - 1);
  }
}
__device__ __forceinline__ bool holds_id(const int* set, int slots, int id)
{
  unsigned h = (static_cast<unsigned>(id) * kIdHash) & (slots - 1);
  for (int p = 0; p < slots; p++) {
    const int t = set[h];
    if (t == -1) return false;
    if (t == id) return true;
    h = (h + 1) & (slots - 1);
  }
  return false;
}

/// (distance bits << 32) | id: the total order of every kept list (search_kernels.cuh:365-368).
__device__ __forceinline__ unsigned long long rank_key(float d, unsigned id)
{
  return (static_cast<unsigned long long>(__float_as_uint(d)) << 32) | id;
}

/// Ascending bitonic sort of P (power of two) 64-bit keys in shared memory.
__device__ __forceinline__ void bitonic_sort(unsigned long long* key, int P)
{
  for (int size = 2; size <= P; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int i = threadIdx.x; i < P; i += blockDim.x) {
        const int j = i ^ stride;
        if (j > i) {
          const bool up              = (i & size) == 0;
          const unsigned long long a = key[i], b = key[j];
          if ((a > b) == up) {
            key[i] = b;
            key[j] = a;
          }
        }
      }
      __syncthreads();
    }
  }
}

/// The key of a lane after it met the one `stride` lanes off: the smaller or the larger of the two.
__device__ __forceinline__ unsigned long long met(unsigned long long mine, int stride, bool smaller)
{
  const unsigned long long other = __shfl_xor_sync(0xffffffffu, mine, stride);
  return (mine < other) == smaller ? mine : other;
}

/// src[0, count) and kNoKey up to `width` (a power of two, 64 at least) in ascending order into key [width], another
/// array: the network of bitonic_sort with 64 keys to a warp, two a lane, so that the steps of 32 places and fewer of a
/// size take one barrier together (512 keys: 10 barriers, where one after every step is 45). All threads of the block
/// call it.
__device__ __forceinline__ void sort_keys(const unsigned long long* src, int count, unsigned long long* key, int width)
{
  const int lane = threadIdx.x & 31, warp0 = (threadIdx.x >> 5) * 64, all = blockDim.x * 2;
  auto finish    = [&](unsigned long long& lo, unsigned long long& hi, bool up) {  // steps of 32 to 1
    const bool keep               = (lo < hi) == up;
    const unsigned long long less = keep ? lo : hi;
    hi                            = keep ? hi : lo;
    lo                            = less;
#pragma unroll 1
    for (int stride = 16; stride > 0; stride >>= 1) {
      const bool smaller = ((lane & stride) == 0) == up;
      lo                 = met(lo, stride, smaller);
      hi                 = met(hi, stride, smaller);
    }
  };
  for (int at = warp0 + lane; at < width; at += all) {
    unsigned long long lo = at < count ? src[at] : kNoKey, hi = at + 32 < count ? src[at + 32] : kNoKey;
#pragma unroll 1
    for (int size = 2; size <= 32; size <<= 1)
#pragma unroll 1
      for (int stride = size >> 1; stride > 0; stride >>= 1) {
        const bool first = (lane & stride) == 0;
        lo               = met(lo, stride, first == ((at & size) == 0));
        hi               = met(hi, stride, first == (((at + 32) & size) == 0));
      }
    finish(lo, hi, (at & 64) == 0);
    key[at]      = lo;
    key[at + 32] = hi;
  }
  __syncthreads();
  for (int size = 128; size <= width; size <<= 1) {
    for (int stride = size >> 1; stride >= 64; stride >>= 1) {
      for (int p = threadIdx.x; p < width / 2; p += blockDim.x) {
        const int i                = 2 * p - (p & (stride - 1));
        const unsigned long long a = key[i], b = key[i + stride];
        if ((a > b) == ((i & size) == 0)) {
          key[i]          = b;
          key[i + stride] = a;
        }
      }
      __syncthreads();
    }
    for (int at = warp0 + lane; at < width; at += all) {
      unsigned long long lo = key[at], hi = key[at + 32];
      finish(lo, hi, (at & size) == 0);
      key[at]      = lo;
      key[at + 32] = hi;
    }
    __syncthreads();
  }
}

struct radix_cut_t {
  unsigned long long prefix, mask;
};

/// Threshold of the R smallest of n distinct 64-bit keys (n > R): 8-bit radix passes from the top
/// bits, stopping at the first pass whose bucket is taken whole. On return exactly R keys k satisfy
/// (k & mask) <= prefix. hi_at(i) / lo_at(i) give the two 32-bit words of key i; the passes over
/// the high word (the distance) never touch the low one (the id), which only breaks ties. All
/// threads of the block call it.
template <typename HiAt, typename LoAt>
__device__ __forceinline__ radix_cut_t radix_cut(HiAt hi_at, LoAt lo_at, int n, int R, unsigned* hist,
                                                 int* ctrl)
{
  unsigned prefix_hi = 0u, mask_hi = 0u, prefix_lo = 0u, mask_lo = 0u;
  int need = R;
  for (int pass = 0; pass < 8; pass++) {
    const int word = pass < 4 ? 1 : 0, shift = 24 - 8 * (pass & 3);
    for (int i = threadIdx.x; i < 256; i += blockDim.x)
      hist[i] = 0;
    __syncthreads();
    if (word == 1) {
      for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const unsigned h = hi_at(i);
        if ((h & mask_hi) == prefix_hi) atomicAdd(&hist[(h >> shift) & 255], 1u);
      }
    } else {
      for (int i = threadIdx.x; i < n; i += blockDim.x) {
        if (hi_at(i) != prefix_hi) continue;
        const unsigned l = lo_at(i);
        if ((l & mask_lo) == prefix_lo) atomicAdd(&hist[(l >> shift) & 255], 1u);
      }
    }
    __syncthreads();
    if (threadIdx.x < 32) {
      // lane l owns digits 8l .. 8l+7: the digit at which the running count reaches `need`
      const int lane = threadIdx.x;
      unsigned h[8], mine = 0;
#pragma unroll
      for (int t = 0; t < 8; t++) {
        h[t] = hist[8 * lane + t];
        mine += h[t];
      }
      unsigned inc = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += u;
      }
      const unsigned before = inc - mine;
      if (before < static_cast<unsigned>(need) && inc >= static_cast<unsigned>(need)) {
        unsigned cum = before, size = h[7];
        int d        = 7;
#pragma unroll
        for (int t = 0; t < 8; t++) {
          if (cum + h[t] >= static_cast<unsigned>(need)) {
            d    = t;
            size = h[t];
            break;
          }
          cum += h[t];
        }
        ctrl[kBin]  = 8 * lane + d;                  // digit
        ctrl[kLeft] = need - static_cast<int>(cum);  // still needed from that bucket
        ctrl[kSize] = static_cast<int>(size);        // bucket size
      }
    }
    __syncthreads();
    const int digit = ctrl[kBin], left = ctrl[kLeft], bucket = ctrl[kSize];
    if (word == 1) {
      prefix_hi |= static_cast<unsigned>(digit) << shift;
      mask_hi |= 255u << shift;
    } else {
      prefix_lo |= static_cast<unsigned>(digit) << shift;
      mask_lo |= 255u << shift;
    }
    need = left;
    __syncthreads();
    if (bucket == left) break;
  }
  return radix_cut_t{(static_cast<unsigned long long>(prefix_hi) << 32) | prefix_lo,
                     (static_cast<unsigned long long>(mask_hi) << 32) | mask_lo};
}

/// What a selection expects: counters at zero, no range yet. A barrier belongs behind it.
__device__ __forceinline__ void selection_begin(unsigned* hist, int* ctrl)
{
  for (int i = threadIdx.x; i < 256; i += blockDim.x)
    hist[i] = 0;
  if (threadIdx.x == 0) {
    ctrl[kEmitted] = 0;
    ctrl[kSide]    = 0;
    ctrl[kLow]     = -1;
    ctrl[kHigh]    = 0;
  }
}

/// The range of the high words of n keys, in ctrl[kLow] and ctrl[kHigh]. After selection_begin and a barrier;
/// ends in one.
template <typename HiAt>
__device__ __forceinline__ void find_range(HiAt hi_at, int n, int* ctrl)
{
  unsigned low = ~0u, high = 0u;
#pragma unroll 4
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const unsigned h = hi_at(i);
    low              = min(low, h);
    high             = max(high, h);
  }
  low  = __reduce_min_sync(0xffffffffu, low);
  high = __reduce_max_sync(0xffffffffu, high);
  if ((threadIdx.x & 31) == 0 && low <= high) {
    atomicMin(reinterpret_cast<unsigned*>(&ctrl[kLow]), low);
    atomicMax(reinterpret_cast<unsigned*>(&ctrl[kHigh]), high);
  }
  __syncthreads();
}

/// emit(high word, low word) for the R smallest of n distinct keys (n > R), in any order; hi_at(i) /
/// lo_at(i) give the two words of key i. The high words (distances of one query: a narrow range of bit
/// patterns, known to be [ctrl[kLow], ctrl[kHigh]]) are counted in 256 bins over their range, the bin
/// that holds the R-th key is found, and a second pass takes what lies below it and puts the bin's own
/// members aside, which are ranked among themselves. With more than 128 of those (many equal or nearly
/// equal distances) radix_cut finds the threshold. With the range three passes over the keys and five
/// barriers; passes of their own for the members and the taking made it four and nine. hist: 256 words,
/// counters and then the members. After selection_begin and find_range; all threads of the block call it,
/// and a barrier belongs behind it.
template <typename HiAt, typename LoAt, typename Emit>
__device__ __forceinline__ void take_smallest(HiAt hi_at, LoAt lo_at, int n, int R, unsigned* hist, int* ctrl, Emit emit)
{
  constexpr unsigned kSideRoom = 128;
  const unsigned lo = static_cast<unsigned>(ctrl[kLow]), hi = static_cast<unsigned>(ctrl[kHigh]);
  const int sh = max(0, 24 - __clz(static_cast<int>(hi - lo)));  // (hi - lo) >> sh < 256
  for (int i = threadIdx.x; i < n; i += blockDim.x)
    atomicAdd(&hist[(hi_at(i) - lo) >> sh], 1u);
  __syncthreads();
  if (threadIdx.x < 32) {
    // lane l owns bins 8l .. 8l+7: the bin at which the running count reaches R
    const int lane = threadIdx.x;
    unsigned h[8], mine = 0;
#pragma unroll
    for (int t = 0; t < 8; t++) {
      h[t] = hist[8 * lane + t];
      mine += h[t];
    }
    unsigned inc = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned u = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += u;
    }
    const unsigned before = inc - mine;
    if (before < static_cast<unsigned>(R) && inc >= static_cast<unsigned>(R)) {
      unsigned cum = before, size = h[7];
      int d        = 7;
#pragma unroll
      for (int t = 0; t < 8; t++) {
        if (cum + h[t] >= static_cast<unsigned>(R)) {
          d    = t;
          size = h[t];
          break;
        }
        cum += h[t];
      }
      ctrl[kBin]  = 8 * lane + d;
      ctrl[kLeft] = R - static_cast<int>(cum);
      ctrl[kSize] = static_cast<int>(size);
    }
  }
  __syncthreads();
  const unsigned bin  = static_cast<unsigned>(ctrl[kBin]);
  const unsigned left = static_cast<unsigned>(ctrl[kLeft]), size = static_cast<unsigned>(ctrl[kSize]);
  if (left < size && size > kSideRoom) {
    const radix_cut_t c = radix_cut(hi_at, lo_at, n, R, hist, ctrl);
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const unsigned h = hi_at(i), l = lo_at(i);
      if ((((static_cast<unsigned long long>(h) << 32) | l) & c.mask) <= c.prefix) emit(h, l);
    }
    return;
  }
  unsigned long long* side = reinterpret_cast<unsigned long long*>(hist);  // the counters are dead
  const unsigned taken     = left == size ? bin + 1 : bin;                // the bins below are taken whole
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const unsigned h = hi_at(i), b = (h - lo) >> sh;
    if (b < taken)
      emit(h, lo_at(i));
    else if (b == bin)
      side[atomicAdd(&ctrl[kSide], 1)] = (static_cast<unsigned long long>(h) << 32) | lo_at(i);
  }
  if (left == size) return;
  __syncthreads();
  if (threadIdx.x < size) {
    const unsigned long long mine = side[threadIdx.x];
    unsigned below                = 0;
    for (unsigned j = 0; j < size; j++)
      below += side[j] < mine;
    if (below < left) emit(static_cast<unsigned>(mine >> 32), static_cast<unsigned>(mine));
  }
}

/// The `want` smallest of cnt distinct keys src[0, cnt) into dst (another array), ascending: a group of
/// lanes counts the keys below its own and puts it there. No step depends on another, which suits the
/// short lists a merge usually sorts better than a sorting network run by one warp. A lane counts eight keys at
/// least: with 32 lanes for each of 32 keys a merge of 1 024 threads took 3.3 thousand cycles, with four 2.8. One
/// lane a key has a loop of its own, which reads two keys a load: 7 499 queries whose first round keeps 128 of 128
/// keys, when those were ranked, 303 us without it, 293 with it; 10 000 with default parameters 2 322 and 2 277.
/// cnt <= blockDim.x.
__device__ __forceinline__ void rank_sort(const unsigned long long* src, int cnt, unsigned long long* dst, int want)
{
  int lanes = 1;  // per key
  while (cnt > 8 * lanes && 2 * lanes * cnt <= static_cast<int>(blockDim.x))
    lanes *= 2;
  const int at = threadIdx.x / lanes, sub = threadIdx.x & (lanes - 1);
  if ((threadIdx.x & ~31u) / lanes >= static_cast<unsigned>(cnt)) return;  // a warp without a key
  const unsigned long long mine = src[min(at, cnt - 1)];
  int below                     = 0;
  if (lanes == 1) {
#pragma unroll 8
    for (int j = 0; j < cnt; j++)
      below += src[j] < mine;
  } else {
#pragma unroll 4
    for (int j = sub; j < cnt; j += lanes)
      below += src[j] < mine;
    for (int o = 1; o < lanes; o <<= 1)
      below += __shfl_xor_sync(0xffffffffu, below, o);
  }
  if (sub == 0 && at < cnt && below < want) dst[below] = mine;
}

constexpr int kCounted = 128;  // new keys whose places are counted at most (see merge_sorted)

/// The first `want` keys of the ascending list old[0, n) and the m distinct keys add[0, m), none of them in
/// the list, into dst, ascending; order [m] is scratch. A new key's place is the number of new keys below
/// it, counted, and of old ones, found by halving; an old key's is its own plus the new ones below it,
/// halving in their order. One barrier where a sorting network over all of them, with one after every step, has 36
/// (256 keys) to 55 (1 024 keys). Counting is quadratic in the new keys: more than kCounted the caller has put into
/// ascending order (sort_keys, with barriers of its own). us a search with all places counted, and with kCounted of 64,
/// 128 and 256: 1 000 queries, 512 kept and 512 reranked rows 1 470, 1 427, 1 429 and 1 424; 2 000, 256 and 256 1 550, 1 541, 1 544 and
/// 1 553; 2 500 ranked by sketch distance into 512 3 265, 3 154, 3 154 and 3 158. All threads of the block call it.
__device__ __forceinline__ void merge_sorted(const unsigned long long* old, int n, const unsigned long long* add, int m,
                                             unsigned long long* order, int want, unsigned long long* dst)
{
  auto below = [](const unsigned long long* list, int count, unsigned long long key) {
    int lo = 0, hi = count;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (list[mid] < key)
        lo = mid + 1;
      else
        hi = mid;
    }
    return lo;
  };
  if (m > kCounted) {
    for (int j = threadIdx.x; j < m; j += blockDim.x) {
      const int place = j + below(old, n, order[j]);
      if (place < want) dst[place] = order[j];
    }
  } else {
    for (int j = threadIdx.x; j < m; j += blockDim.x) {
      const unsigned long long mine = add[j];
      int at                        = 0;
#pragma unroll 4
      for (int i = 0; i < m; i++)
        at += add[i] < mine;
      order[at]       = mine;
      const int place = at + below(old, n, mine);
      if (place < want) dst[place] = mine;
    }
    __syncthreads();
  }
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const unsigned long long mine = old[i];
    const int place               = i + below(order, m, mine);
    if (place < want) dst[place] = mine;
  }
}

/// float(h) - q for an fp16 bit pattern h: the mixed-precision subtract of sm_100 (PTX ISA 8.6),
/// the same value as converting first (the conversion is exact) without the conversion.
__device__ __forceinline__ float half_minus(unsigned short h, float q)
{
  float d;
  asm("sub.rn.f32.f16 %0, %1, %2;" : "=f"(d) : "h"(h), "f"(q));
  return d;
}

/// Row `id` of an array with `width` elements per row: behind `base`, or (kDealt and a table given)
/// in the memory of the GPU that holds its range (search_kernels.cuh:40-55).
template <bool kDealt, typename T>
__device__ __forceinline__ const T* row_of(const T* base, const row_map& m, int id, int width)
{
  if constexpr (kDealt) {
    if (m.ptrs != nullptr) {
      const int g = id / m.rows;
      return reinterpret_cast<const T*>(m.ptrs[g]) + static_cast<int64_t>(id - g * m.rows) * width;
    }
  }
  return base + static_cast<int64_t>(id) * width;
}

/// Rows that may sit in another GPU's memory are not prefetched into this GPU's L2.
template <bool kDealt>
__device__ __forceinline__ bool may_prefetch(const row_map& m)
{
  return !kDealt || m.ptrs == nullptr;
}

/// The query's side of the sketch distance, made once per query block by its first warp.
/// The reference scores sum_k (c_k s_k - q_k)^2 in fp32 per candidate (search_kernels.cuh:228-251).
/// Expanded: sum_k (c_k s_k)^2 - 2 sum_k c_k (s_k q_k) + sum_k q_k^2. The first sum is a constant
/// of the row, computed when the index is placed (norm [n]); the last is a constant of the
/// query; the middle one becomes an exact integer dot product of the int8 codes with 16-bit weights
/// w_k = rint(s_k q_k / alpha), alpha = max_k |s_k q_k| / 32000 (two codes per dp2a). The value
/// differs from the fp32 sum by the rounding of the weights (at most 1.6e-5 of the largest product
/// per term) and of three fp32 operations. Every operation and its order are stated here and in
/// the CPU checker, which evaluates the same form.
/// Writes w16 [S / 2] (weights of codes 2i and 2i + 1 in the low and high half of word i) and
/// kq[0] = -2 alpha, kq[1] = sum_k q_k^2 (partial sum k mod 32, butterfly with strides 1 .. 16).
__device__ __forceinline__ void sketch_query_setup(const float* __restrict__ qs, const float* __restrict__ scale,
                                                   int S, int* w16, float* kq)
{
  const int lane = threadIdx.x & 31;
  float amax = 0.f, qq = 0.f;
  for (int k = lane; k < S; k += 32) {
    const float q = qs[k];
    amax          = fmaxf(amax, fabsf(__fmul_rn(scale[k], q)));
    qq            = __fmaf_rn(q, q, qq);
  }
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    qq   = __fadd_rn(qq, __shfl_xor_sync(0xffffffffu, qq, o));
  }
  const float alpha = (amax > 0.f && amax <= FLT_MAX) ? __fdiv_rn(amax, 32000.0f) : 1.0f;
  short* w = reinterpret_cast<short*>(w16);
  for (int k = lane; k < S; k += 32) {
    const float r = rintf(__fdiv_rn(__fmul_rn(scale[k], qs[k]), alpha));
    w[k]          = static_cast<short>(r != r ? 0 : static_cast<int>(fminf(fmaxf(r, -32000.0f), 32000.0f)));
  }
  if (lane == 0) {
    kq[0] = -2.0f * alpha;
    kq[1] = qq;
  }
}

/// Sketch distances of the candidates cand[0, n) into dist[0, n): kLw (a power of two >= S / 16)
/// lanes own a row, sixteen codes (one 16-byte load) and their eight weight pairs each; a lane's
/// dot product takes eight dp2a; the lanes of a row add theirs by a butterfly; four rows per lane
/// group are in flight. A lane past the last row works on the last row and a lane past the last
/// chunk on chunk 0 with zero weights; their results are dropped or add 0.
// ---- L2 residency ---------------------------------------------------------------------------------
//
// The int8 sketch and its row constants are the arrays every query reads most often (hundreds of
// rows per round) and, for an index of a million rows, small enough to stay in the 126 MB L2 cache
// next to everything else; the fp16 vectors, the lists and the neighbor table are read once or a
// few times per batch and are many times larger. When the host finds that the sketch fits
// (keep_sketch), the first round loads sketch rows and constants with an evict-last policy, and every
// round the lists and the table with an evict-first policy, so that the streaming reads do not push
// the sketch out; the fp16 rows go first too where a large sketch needs the room (pass_vectors).

__device__ __forceinline__ unsigned long long l2_policy_keep()
{
  unsigned long long p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}

__device__ __forceinline__ unsigned long long l2_policy_stream()
{
  unsigned long long p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}

__device__ __forceinline__ uint4 ldg16_hint(const void* a, unsigned long long policy)
{
  uint4 v;
  asm volatile("ld.global.nc.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(a), "l"(policy));
  return v;
}

__device__ __forceinline__ float ldg_f32_hint(const float* a, unsigned long long policy)
{
  float v;
  asm volatile("ld.global.nc.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(a), "l"(policy));
  return v;
}

__device__ __forceinline__ int ldg_i32_hint(const int* a, unsigned long long policy)
{
  int v;
  asm volatile("ld.global.nc.L2::cache_hint.s32 %0, [%1], %2;" : "=r"(v) : "l"(a), "l"(policy));
  return v;
}

template <int kLw, bool kDealt>
__device__ __forceinline__ void sketch_rows_int(const int* cand, int n, const signed char* __restrict__ sketch,
                                                const float* __restrict__ norm, const row_map& map, int S,
                                                const int* w16, const float* kq, float* dist, bool keep)
{
  constexpr int kG = 32 / kLw;  // rows per warp and step
  constexpr int kU = 4;          // rows of a lane group in flight
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int sub = lane % kLw, grp = lane / kLw;
  const bool live  = 16 * sub < S;
  const int subc   = live ? sub : 0;
  int w[8];
  {
    const int4 w0 = reinterpret_cast<const int4*>(w16)[2 * subc];
    const int4 w1 = reinterpret_cast<const int4*>(w16)[2 * subc + 1];
    w[0] = w0.x, w[1] = w0.y, w[2] = w0.z, w[3] = w0.w, w[4] = w1.x, w[5] = w1.y, w[6] = w1.z, w[7] = w1.w;
#pragma unroll
    for (int b = 0; b < 8; b++)
      if (!live) w[b] = 0;
  }
  const float beta = kq[0], qq = kq[1];
  const unsigned long long pol = l2_policy_keep();
  const int rpp = nw * kG;  // rows per step of the block
  for (int jb = 0; jb < n; jb += kU * rpp) {
    uint4 c[kU];
    float nrm[kU];
    int j[kU];
#pragma unroll
    for (int u = 0; u < kU; u++) {
      j[u]            = jb + u * rpp + warp * kG + grp;
      const int id    = cand[min(j[u], n - 1)];
      const uint4* row = reinterpret_cast<const uint4*>(row_of<kDealt>(sketch, map, id, S)) + subc;
      if (keep) {
        c[u]   = ldg16_hint(row, pol);
        nrm[u] = ldg_f32_hint(norm + id, pol);
      } else {
        c[u]   = __ldg(row);
        nrm[u] = __ldg(norm + id);
      }
    }
#pragma unroll
    for (int u = 0; u < kU; u++) {
      int d = __dp2a_lo(w[0], static_cast<int>(c[u].x), 0);
      d     = __dp2a_hi(w[1], static_cast<int>(c[u].x), d);
      d     = __dp2a_lo(w[2], static_cast<int>(c[u].y), d);
      d     = __dp2a_hi(w[3], static_cast<int>(c[u].y), d);
      d     = __dp2a_lo(w[4], static_cast<int>(c[u].z), d);
      d     = __dp2a_hi(w[5], static_cast<int>(c[u].z), d);
      d     = __dp2a_lo(w[6], static_cast<int>(c[u].w), d);
      d     = __dp2a_hi(w[7], static_cast<int>(c[u].w), d);
#pragma unroll
      for (int o = 1; o < kLw; o <<= 1)
        d += __shfl_xor_sync(0xffffffffu, d, o);
      if (j[u] < n && sub == 0)
        dist[j[u]] = fmaxf(__fadd_rn(nrm[u], __fmaf_rn(beta, static_cast<float>(d), qq)), 0.f);
    }
  }
}

/// Eight int8 codes (two 32-bit words) against eight (scale, query) pairs: sum of
/// (code * scale - q)^2 with two fused multiply-adds per code, in code order. The int8 -> float
/// conversion: one byte permute makes the fp16 patterns 0x64bb = 1024 + (code + 128) of two codes,
/// and the mixed-precision subtract of 1152 gives each code exactly, off the conversion pipe.
__device__ __forceinline__ float sketch_chunk8(unsigned w0, unsigned w1, const float* s, const float* q)
{
  const unsigned x0 = w0 ^ 0x80808080u, x1 = w1 ^ 0x80808080u;  // code + 128 in every byte
  float d           = 0.f;
#pragma unroll
  for (int p = 0; p < 4; p++) {
    const unsigned hh = __byte_perm(p < 2 ? x0 : x1, 0x64646464u, (p & 1) ? 0x4342 : 0x4140);
    const float c0    = half_minus(static_cast<unsigned short>(hh & 0xffffu), 1152.0f);
    const float c1    = half_minus(static_cast<unsigned short>(hh >> 16), 1152.0f);
    const float t0    = __fmaf_rn(c0, s[2 * p], -q[2 * p]);
    d                 = __fmaf_rn(t0, t0, d);
    const float t1    = __fmaf_rn(c1, s[2 * p + 1], -q[2 * p + 1]);
    d                 = __fmaf_rn(t1, t1, d);
  }
  return d;
}

/// Two fp32 values side by side.
using f32_two = unsigned long long;
__device__ __forceinline__ f32_two two_of(float a, float b)
{
  f32_two r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}

/// Sixteen int8 codes: sketch_chunk8 of either eight, side by side in packed multiply-adds, then the sum of the two.
/// s [8] and minus_q [8]: scale and negated query value of codes i and 8 + i.
__device__ __forceinline__ float sketch_chunk16(const uint4& w, const f32_two* s, const f32_two* minus_q)
{
  const unsigned x[4] = {w.x ^ 0x80808080u, w.y ^ 0x80808080u, w.z ^ 0x80808080u, w.w ^ 0x80808080u};  // code + 128
  f32_two d           = 0;
#pragma unroll
  for (int p = 0; p < 4; p++) {
    const unsigned two = (p & 1) ? 0x4342 : 0x4140;
    const unsigned a   = __byte_perm(x[p < 2 ? 0 : 1], 0x64646464u, two);
    const unsigned b   = __byte_perm(x[p < 2 ? 2 : 3], 0x64646464u, two);
    const f32_two c0   = two_of(half_minus(static_cast<unsigned short>(a & 0xffffu), 1152.0f),
                                half_minus(static_cast<unsigned short>(b & 0xffffu), 1152.0f));
    const f32_two c1   = two_of(half_minus(static_cast<unsigned short>(a >> 16), 1152.0f),
                                half_minus(static_cast<unsigned short>(b >> 16), 1152.0f));
    f32_two t;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(t) : "l"(c0), "l"(s[2 * p]), "l"(minus_q[2 * p]));
    asm("fma.rn.f32x2 %0, %1, %1, %2;" : "=l"(d) : "l"(t), "l"(d));
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(t) : "l"(c1), "l"(s[2 * p + 1]), "l"(minus_q[2 * p + 1]));
    asm("fma.rn.f32x2 %0, %1, %1, %2;" : "=l"(d) : "l"(t), "l"(d));
  }
  float d0, d1;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d0), "=f"(d1) : "l"(d));
  return __fadd_rn(d0, d1);
}

/// The sketch distance in the reference's own fp32 terms, sum_k (c_k s_k - q_k)^2
/// (search_kernels.cuh:228-251), for the waves: there a candidate's row arrives from memory later
/// than the arithmetic on it takes, so the form that needs nothing but the row (no row constant)
/// is the faster one; the first round, whose rows are mostly in the L2 cache already, is bound by
/// instructions and takes the integer form above. Summation order (shared with the CPU checker):
/// chunk c of 8 codes is partial sum c (two fused multiply-adds per code, in code order), a
/// butterfly over the next power of two >= S / 8 partial sums with strides 1, 2, 4, ... A lane
/// holds two neighbouring chunks (one 16-byte load) and adds them itself (stride 1); kLw (a power
/// of two >= S / 16) lanes own a row; two rows per lane group are in flight. A lane past the last
/// chunk works on chunk 0 with scales and query 0 and adds exactly 0.
/// kPaired: the two chunks of a lane in packed operations, half as many to issue, for the waves (us a search, one by one
/// and packed: three waves of 16 384 entries 7 992 and 7 869, of 32 768 ranked by sketch distance 3 429 and 3 334, of 4 096
/// 1 807 and 1 734, 10 000 tuned 835 and 829, 1 000 with default parameters 291 and 287). First rounds that rank by
/// sketch distance spill with it: 355 and 366.
template <int kLw, bool kDealt, bool kPaired>
__device__ __forceinline__ void sketch_rows_f32(const int* cand, int n, const signed char* __restrict__ sketch,
                                                const row_map& map, int S, const float* sc, const float* qv,
                                                float* dist)
{
  constexpr int kG = 32 / kLw;  // rows per warp and step
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int sub = lane % kLw, grp = lane / kLw;
  const bool live = 16 * sub < S;
  const int subc  = live ? sub : 0;
  // the lane's sixteen scales and query values, 16 bytes at a time (both arrays start on 16-byte
  // boundaries): a quarter of the shared-memory traffic of single words
  float cs[16], cq[16];
#pragma unroll
  for (int b = 0; b < 4; b++) {
    const float4 s4 = live ? reinterpret_cast<const float4*>(sc + sub * 16)[b] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 q4 = live ? reinterpret_cast<const float4*>(qv + sub * 16)[b] : make_float4(0.f, 0.f, 0.f, 0.f);
    cs[4 * b] = s4.x, cs[4 * b + 1] = s4.y, cs[4 * b + 2] = s4.z, cs[4 * b + 3] = s4.w;
    cq[4 * b] = q4.x, cq[4 * b + 1] = q4.y, cq[4 * b + 2] = q4.z, cq[4 * b + 3] = q4.w;
  }
  f32_two s2[8], q2[8];
#pragma unroll
  for (int i = 0; i < 8; i++) {
    s2[i] = two_of(cs[i], cs[8 + i]);
    q2[i] = two_of(-cq[i], -cq[8 + i]);
  }
  const int rpp = nw * kG;  // rows per step of the block
  if (n <= 0) return;
  // The ids of a step come in behind the step before: where they are in global memory they took a third of a
  // step's time (three waves of 16 384 entries: 178 and 149 thousand cycles of scoring, 8 582 and 8 287 us a
  // search). The rows a step ahead as well: no faster (8 316).
  int id[2];
#pragma unroll
  for (int u = 0; u < 2; u++)
    id[u] = cand[min(u * rpp + warp * kG + grp, n - 1)];
  for (int jb = 0; jb < n; jb += 2 * rpp) {
    uint4 w[2];
    int j[2];
#pragma unroll
    for (int u = 0; u < 2; u++) {
      j[u] = jb + u * rpp + warp * kG + grp;
      w[u] = __ldg(reinterpret_cast<const uint4*>(row_of<kDealt>(sketch, map, id[u], S)) + subc);
    }
#pragma unroll
    for (int u = 0; u < 2; u++)
      id[u] = cand[min(j[u] + 2 * rpp, n - 1)];
#pragma unroll
    for (int u = 0; u < 2; u++) {
      float d;
      if constexpr (kPaired)
        d = sketch_chunk16(w[u], s2, q2);
      else
        d = __fadd_rn(sketch_chunk8(w[u].x, w[u].y, cs, cq), sketch_chunk8(w[u].z, w[u].w, cs + 8, cq + 8));
#pragma unroll
      for (int o = 1; o < kLw; o <<= 1)
        d = __fadd_rn(d, __shfl_xor_sync(0xffffffffu, d, o));
      if (j[u] < n && sub == 0) dist[j[u]] = d;
    }
  }
}

/// Where element i of the query sits in shared memory for exact_pair: within every step of 64
/// elements the 16-byte chunks are dealt so that the eight lanes of a row group read consecutive
/// chunks with each of their two loads (chunks 0, 2, 4, ... first, then 1, 3, 5, ...): one
/// wavefront per load instead of two. The array takes the dimension rounded up to 64 floats.
__device__ __forceinline__ int query_slot(int i)
{
  const int chunk = (i & 63) >> 2;
  return (i & ~63) + ((((chunk & 1) << 3) + (chunk >> 1)) << 2) + (i & 3);
}

/// Rows j and j + stride of a lane group: squared distances of two fp16 rows to the query fq (laid
/// out by query_slot)
/// (shared memory, read 16 bytes at a time).
/// Both row pointers are valid (a row that is not wanted is replaced by any row by the caller, who
/// drops the result). kMode 0: any D that is a multiple of 8; 1: D a multiple of 128, so no step
/// needs a bounds check; 2: D = 128, one step with constant offsets. kPass: the rows leave the L2 cache first.
template <int kMode, bool kPass>
__device__ __forceinline__ void exact_pair(const uint4* const (&row)[2], int Drt, int sub, const float* fq,
                                           float (&out)[2])
{
  constexpr bool kWhole = kMode != 0;
  const int D           = kMode == 2 ? 128 : Drt;
  // (The policy is made at each load: held in two registers over the loop it is no faster at 128 dimensions, 1 074 and
  // 1 076 us a search, and slower at others: 32 dimensions 920 and 935, 64 1 007 and 1 026, 256 1 472 and 1 487.)
  float acc[2][4];
#pragma unroll
  for (int u = 0; u < 2; u++)
#pragma unroll
    for (int t = 0; t < 4; t++)
      acc[u][t] = 0.f;
  // two 16-byte steps of both rows are loaded before any of them is used
  for (int h0 = 8 * sub; h0 < D; h0 += 128) {
    uint4 v[2][2];
#pragma unroll
    for (int s = 0; s < 2; s++)
#pragma unroll
      for (int u = 0; u < 2; u++)
        if (kWhole || h0 + 64 * s < D) {
          const uint4* at = row[u] + ((h0 + 64 * s) >> 3);
          v[s][u]         = kPass ? ldg16_hint(at, l2_policy_stream()) : __ldg(at);
        }
#pragma unroll
    for (int s = 0; s < 2; s++) {
      const int hs = h0 + 64 * s;
      if (kWhole || hs < D) {
        const float4 q0 = *reinterpret_cast<const float4*>(fq + (hs - 8 * sub) + 4 * sub);
        const float4 q1 = *reinterpret_cast<const float4*>(fq + (hs - 8 * sub) + 4 * sub + 32);
        const float qq[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
#pragma unroll
        for (int u = 0; u < 2; u++) {
          const unsigned h2[4] = {v[s][u].x, v[s][u].y, v[s][u].z, v[s][u].w};
#pragma unroll
          for (int t = 0; t < 4; t++) {
            const float a = half_minus(static_cast<unsigned short>(h2[t] & 0xffffu), qq[2 * t]);
            const float b = half_minus(static_cast<unsigned short>(h2[t] >> 16), qq[2 * t + 1]);
            acc[u][t]     = __fmaf_rn(b, b, __fmaf_rn(a, a, acc[u][t]));
          }
        }
      }
    }
  }
  // butterfly over the 32 partial sums, strides 1, 2 (inside the lane), then 4, 8, 16 (lanes)
#pragma unroll
  for (int u = 0; u < 2; u++) {
    float v = __fadd_rn(__fadd_rn(acc[u][0], acc[u][1]), __fadd_rn(acc[u][2], acc[u][3]));
#pragma unroll
    for (int o = 1; o < 8; o <<= 1)
      v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
    out[u] = v;
  }
}

/// Squared distances of the fp16 rows sid[0, ns) (entries < 0 are skipped) to the fp32 query fq,
/// written over sdv. Summation order (shared with the CPU checker): element pair k feeds partial
/// sum k mod 32 with two fused multiply-adds; a butterfly over the 32 partial sums with strides
/// 1, 2, 4, 8, 16 (search_kernels.cuh:325-342 is the reference's warp-per-row form of the same
/// sum). Eight lanes own a row, each reading 16 bytes per step (partial sums 4 lane .. 4 lane + 3);
/// a warp works on eight rows at a time.
template <bool kDealt, int kMode, bool kPass>
__device__ __forceinline__ void exact_rows(const int* sid, int ns, const __half* __restrict__ vectors,
                                           const row_map& map, int Drt, const float* fq, float* sdv)
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int sub = lane & 7, grp = lane >> 3;
  const int D   = kMode == 2 ? 128 : Drt;
  for (int jb = warp * 4 + grp; jb < ns + warp * 4 + grp; jb += nw * 8) {
    int j[2];
    bool wanted[2];
    const uint4* row[2];
#pragma unroll
    for (int u = 0; u < 2; u++) {
      j[u]         = jb + u * nw * 4;
      const int id = j[u] < ns ? sid[j[u]] : -1;
      wanted[u]    = id >= 0;
      // a slot without a row works on a row this GPU holds (cached after its first use) and drops
      // the result
      row[u] = reinterpret_cast<const uint4*>(row_of<kDealt>(vectors, map, wanted[u] ? id : map.local, D));
    }
    float out[2];
    exact_pair<kMode, kPass>(row, D, sub, fq, out);
#pragma unroll
    for (int u = 0; u < 2; u++)
      if (wanted[u] && sub == 0) sdv[j[u]] = out[u];
  }
}

template <bool kDealt, bool kPass>
__device__ __forceinline__ void exact_distances(const int* sid, int ns, const __half* __restrict__ vectors,
                                                const row_map& map, int D, const float* fq, float* sdv)
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (D == 128) {
    exact_rows<kDealt, 2, kPass>(sid, ns, vectors, map, D, fq, sdv);
  } else if ((D & 127) == 0) {
    exact_rows<kDealt, 1, kPass>(sid, ns, vectors, map, D, fq, sdv);
  } else if ((D & 7) == 0) {
    exact_rows<kDealt, 0, kPass>(sid, ns, vectors, map, D, fq, sdv);
  } else {
    for (int j = warp; j < ns; j += nw) {
      if (sid[j] < 0) continue;
      const __half2* row = reinterpret_cast<const __half2*>(row_of<kDealt>(vectors, map, sid[j], D));
      float acc          = 0.f;
      for (int k = lane; k < D / 2; k += 32) {
        const float2 x = __half22float2(row[k]);
        const float a  = __fsub_rn(x.x, fq[2 * k]);
        const float b  = __fsub_rn(x.y, fq[2 * k + 1]);
        acc            = __fmaf_rn(b, b, __fmaf_rn(a, a, acc));
      }
#pragma unroll
      for (int o = 1; o < 32; o <<= 1)
        acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, o));
      if (lane == 0) sdv[j] = acc;
    }
  }
  __syncthreads();
}

/// Merge the new (distance, id) pairs sid / sdv [0, ns) (entries with sid < 0 are skipped; no id is
/// in the kept list already) into the kept list of KO: the KO smallest keys, ascending, padded
/// with (-1, +inf), written to pb / pd. Same result as sorting kept + new and taking the first KO
/// distinct keys (search_kernels.cuh:372-415). A new key beyond the last entry of a full kept list
/// cannot make it and is dropped at once; what remains is sorted directly when it is short, or the
/// KO smallest are selected first. kid / kd: the kept list as it was (shared memory), nk its entries with
/// an id (it is packed: those come first); ctrl[kMerged] is zero. pool holds KO + ns keys, sorted holds
/// 2 * P (P a power of two >= KO). oi / od (k > 0): the first k entries go there too, the results of a
/// last round.
__device__ __forceinline__ void merge_into_kept(unsigned long long* pool,
                                                unsigned long long* sorted,
                                                int P,
                                                long long* pb,
                                                float* pd,
                                                int KO,
                                                const int* kid,
                                                const float* kd,
                                                int nk,
                                                const int* sid,
                                                const float* sdv,
                                                int ns,
                                                unsigned* hist,
                                                int* ctrl,
                                                long long* oi = nullptr,
                                                float* od = nullptr,
                                                int k = 0)
{
  const unsigned long long bound =
    nk == KO && KO > 0 ? rank_key(kd[KO - 1], static_cast<unsigned>(kid[KO - 1])) : kNoKey;
  for (int i = threadIdx.x; i < nk; i += blockDim.x)
    pool[i] = rank_key(kd[i], static_cast<unsigned>(kid[i]));
  for (int i = threadIdx.x; i < ns; i += blockDim.x) {
    if (sid[i] < 0) continue;
    const unsigned long long k = rank_key(sdv[i], static_cast<unsigned>(sid[i]));
    if (k < bound) pool[nk + atomicAdd(&ctrl[kMerged], 1)] = k;
  }
  __syncthreads();
  const int total = nk + ctrl[kMerged];
  const int cnt   = min(total, KO);
  // New keys that fit behind the kept ones go to their places among them. Other short lists are sorted by ranking,
  // at most kRankSteps comparisons a thread, and half of that where KO keys are few of the total, which are
  // rather selected first (always in a block of 128 threads, of which many share a multiprocessor); longer ones by the
  // network. us a search: where the places were left to the ranking whenever that was short enough, and now, 1 000
  // queries with 128 kept and 128 reranked rows 340 and 330, 10 000 2 404 and 2 322, 4 000 wide rows with 256 1 631 and
  // 1 590. Limits of 32, 64 and 128 comparisons: 10 000 queries with 256 kept and 512 reranked rows in three waves 7 606,
  // 7 597 and 7 705 (7 867 with a barrier for every step of the network), 2 000 with 192 and 384 1 396, 1 394 and 1 400
  // (1 428), 148 with 512 and 512 165, 165 and 165 (172). The half, at 32 kept of 300 to 512 reranked rows: 55 queries
  // 126.9 and 123.5, 296 135.6 and 131.5; at 32 of 128 one query takes 66 when it selects first and 63.
  constexpr int kRankSteps = 64;
  const int threads        = blockDim.x;
  const auto few           = [&](int keys, int steps) { return keys <= threads && keys * keys <= steps * threads; };
  const bool places        = nk > 0 && total - nk <= P;
  // what is sorted by the network, if anything (one place in the code for all: every copy of it costs the round's
  // other phases registers)
  const unsigned long long* from = pool;
  unsigned long long* to         = sorted;
  int count = 0, width = P;
  if (places) {
    if (total - nk > kCounted) from = pool + nk, to = sorted + P, count = total - nk, width = 2 * kCounted;
  } else if (total <= 2 * P ? few(total, kRankSteps) : threads > kRoundThreads && few(total, kRankSteps / 2)) {
    rank_sort(pool, total, sorted, KO);
  } else if (total <= 2 * P) {
    count = total;
  } else {
    // the KO smallest are selected first (into the upper half of the sort region), then sorted
    unsigned long long* picked = sorted + max(P, 32);
    auto hi_at                 = [&](int i) { return static_cast<unsigned>(pool[i] >> 32); };
    auto lo_at                 = [&](int i) { return static_cast<unsigned>(pool[i]); };
    selection_begin(hist, ctrl);
    __syncthreads();
    find_range(hi_at, total, ctrl);
    take_smallest(hi_at, lo_at, total, KO, hist, ctrl, [&](unsigned high, unsigned low) {
      const int s = atomicAdd(&ctrl[kEmitted], 1);
      if (s < P) picked[s] = (static_cast<unsigned long long>(high) << 32) | low;
    });
    __syncthreads();
    if (few(KO, kRankSteps)) {
      rank_sort(picked, KO, sorted, KO);
    } else {
      from = picked, count = KO;
    }
  }
  if (count > 0) {
    while (width < count)
      width <<= 1;
    sort_keys(from, count, to, width);
  }
  if (places) merge_sorted(pool, nk, pool + nk, total - nk, sorted + P, KO, sorted);
  __syncthreads();
  for (int i = threadIdx.x; i < KO; i += blockDim.x) {
    const unsigned long long key = i < cnt ? sorted[i] : kNoKey;
    const long long id = key == kNoKey ? -1 : static_cast<long long>(static_cast<unsigned>(key & 0xffffffffULL));
    const float d      = key == kNoKey ? INFINITY : __uint_as_float(static_cast<unsigned>(key >> 32));
    pb[i] = id;
    pd[i] = d;
    if (i < k) {
      oi[i] = id;
      od[i] = d;
    }
  }
}

// kThreads: 128 with eight blocks per multiprocessor when a block's shared memory allows that; a
// round whose hash set is too large for eight blocks runs 256, 512 or 1024 threads per block instead,
// so that the blocks that do fit still bring 32 warps to a multiprocessor, and so does a batch with
// too few queries to fill the multiprocessors with small blocks (round_threads).
//
// kShort: a wave of few entries for few queries (short_wave). A block that is alone on its multiprocessor goes through
// every phase once, and waits for its code more than for anything that code could do side by side: no loads ahead, no
// packed sketch distances, no selection among the candidates that beat a full kept list. us a search of a million rows,
// with the longer code and so: one query, 32 start points of 64 neighbors, one wave 63.8 and 63.1, four 96.4 and 94.8,
// 16 start points and three waves 94.1 and 92.6, eight queries 95.2 and 94.4, two by sketch distance with 16 and two 71.9 and
// 70.6.
template <bool kRows, bool kDealt, int kThreads, bool kShort>
__global__ void __launch_bounds__(kThreads, 1024 / kThreads) round_kernel(const round_args a)
{
  constexpr bool kAhead = kRows && !kShort;
  extern __shared__ __align__(16) int smem[];
  let_next_kernel_start();
  const round_layout lay(a);
  const int q = blockIdx.x;
  int* table  = smem + lay.table;
  int* cand   = a.cand_global ? a.cand_global + static_cast<int64_t>(q) * a.nmax : smem + lay.cand;
  float* dist = a.dist_global ? a.dist_global + static_cast<int64_t>(q) * a.nmax
                              : reinterpret_cast<float*>(smem + lay.dist);
  unsigned long long* pool   = reinterpret_cast<unsigned long long*>(smem + lay.pool);
  unsigned long long* sorted = reinterpret_cast<unsigned long long*>(smem + lay.sorted);
  int* sid                   = smem + lay.sid;
  float* sdv                 = reinterpret_cast<float*>(smem + lay.sdv);
  int* w16                   = smem + lay.qv;
  float* kq                  = reinterpret_cast<float*>(smem + lay.sc);
  float* fq                  = reinterpret_cast<float*>(smem + lay.fq);
  int* st                    = smem + lay.st;
  int* len                   = smem + lay.len;
  unsigned* hist             = reinterpret_cast<unsigned*>(smem + lay.hist);
  int* wsum                  = smem + lay.wsum;
  int* ctrl                  = smem + lay.ctrl;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int S    = a.sw;
  long long* pb  = a.si + static_cast<int64_t>(q) * a.KO;
  float* pd      = a.sd + static_cast<int64_t>(q) * a.KO;

  // The integer form of the sketch distance serves the first round of a search that reranks
  // exactly. Waves take the fp32 sum (see sketch_rows_f32), and so does every round of a search
  // that ranks by sketch distance: there the distances of all rounds meet in one kept list, where
  // an id found twice must bring the same key both times.
  const bool int_form = !kRows && !a.sketch_rank;
  wait_for_previous_kernel();
  if (int_form) {
    if (warp == 0) sketch_query_setup(a.qs + static_cast<int64_t>(q) * S, a.scale, S, w16, kq);
  } else {
    for (int i = threadIdx.x; i < S; i += blockDim.x) {
      reinterpret_cast<float*>(w16)[i] = a.qs[static_cast<int64_t>(q) * S + i];
      kq[i]                            = a.scale[i];
    }
  }
  if (!a.sketch_rank)
    for (int i = threadIdx.x; i < a.D; i += blockDim.x)
      fq[(a.D & 7) ? i : query_slot(i)] = a.Q[static_cast<int64_t>(q) * a.D + i];
  selection_begin(hist, ctrl);
  if (threadIdx.x == 0) {
    ctrl[kDistinct] = 0;
    ctrl[kMerged]   = 0;
    ctrl[kValid]    = 0;
    ctrl[kWithin]   = 0;
  }
  // the kept list as the round finds it (empty in a first round): read once, used by the start points, by
  // the filter of already kept ids and by the merge
  int* kid  = smem + lay.kid;
  float* kd = reinterpret_cast<float*>(smem + lay.kd);
  if constexpr (kRows) {
    for (int i = threadIdx.x; i < a.KO; i += blockDim.x) {
      kid[i] = static_cast<int>(pb[i]);
      kd[i]  = pd[i];
    }
  }

  // cycles per phase of this block (observation only): start points / segments, gather, sketch
  // scoring, selection, filter + prefetch, exact distances, merge
  long long t_prev = 0;
  auto tick = [&](int i) {
    if (a.phase != nullptr && threadIdx.x == 0) {
      const long long t = clock64();
      if (i >= 0) a.phase[static_cast<int64_t>(q) * 8 + i] += t - t_prev;
      t_prev = t;
    }
  };
  tick(-1);
  int total = 0, nseg = a.nseg;
  if constexpr (kRows) {
    // start points: the first nseg kept entries that no earlier wave expanded
    // (search_kernels.cuh:571-631); earlier start points, if there are any, go through a hash set in the
    // table region
    int* pdone       = a.done + static_cast<int64_t>(q) * a.done_stride;
    const bool again = a.done_off > 0;
    if (again)
      for (int i = threadIdx.x; i < a.pick_slots; i += blockDim.x)
        table[i] = -1;
    __syncthreads();
    if (again)
      for (int i = threadIdx.x; i < a.done_off; i += blockDim.x)
        insert_id(table, a.pick_slots, pdone[i]);
    for (int i = threadIdx.x; i < a.KO; i += blockDim.x)
      if (kid[i] >= 0 && (i + 1 == a.KO || kid[i + 1] < 0)) ctrl[kValid] = i + 1;
    if (again) __syncthreads();
    const int per       = (a.KO + kThreads - 1) / kThreads;
    const int i0        = threadIdx.x * per;
    unsigned fresh_bits = 0;
    int mine            = 0;
    for (int i = i0; i < min(a.KO, i0 + per); i++) {
      const int v = kid[i];
      const bool f = v >= 0 && !(again && holds_id(table, a.pick_slots, v));
      if (f) {
        fresh_bits |= 1u << (i - i0);
        mine++;
      }
    }
    int nfresh = 0;
    int at     = block_scan<kThreads>(mine, wsum, nfresh);
    for (int i = i0; i < min(a.KO, i0 + per); i++)
      if (fresh_bits & (1u << (i - i0))) {
        if (at < a.nseg) {
          const int v            = kid[i];
          st[at]                 = v;
          pdone[a.done_off + at] = v;
          // its table row is read next: start bringing it into L2
          if (may_prefetch<kDealt>(a.table_map)) {
            const char* row = reinterpret_cast<const char*>(a.table + static_cast<int64_t>(v) * a.table_len);
            for (int b = 0; b < a.table_len * 4; b += 128)
              asm volatile("prefetch.global.L2 [%0];" ::"l"(row + b));
          }
        }
        at++;
      }
    nseg = min(nfresh, a.nseg);
    for (int o = nseg + threadIdx.x; o < a.nseg; o += blockDim.x)
      pdone[a.done_off + o] = -1;
    total = nseg * a.table_len;
    if (threadIdx.x == 0) ctrl[kStarts] = nseg;
  } else {
    // segment starts and lengths; every segment is either empty or `read` entries long
    int mine = 0;
    for (int c = threadIdx.x; c < a.nseg; c += blockDim.x) {
      const int2 sl = a.seg[static_cast<int64_t>(q) * a.nseg + c];
      st[c]         = sl.x;
      len[c]        = sl.y;
      mine += sl.y;
      if (sl.y > 0) {  // the run of list entries is read next: start bringing it into L2
        const char* run = reinterpret_cast<const char*>(a.lists + static_cast<int64_t>(c) * a.stride + sl.x);
        asm volatile("prefetch.global.L2 [%0];" ::"l"(run));
        asm volatile("prefetch.global.L2 [%0];" ::"l"(run + sl.y * 4 - 4));
      }
    }
    block_scan<kThreads>(mine, wsum, total);
  }

  // distinct ids through an open-addressing hash set (search_kernels.cuh:191-225); a group of lps
  // threads walks one segment, so consecutive threads read consecutive entries, and every thread
  // has four segments' loads in flight before it touches the set
  tick(0);
  const int HT = a.map_words > 0 ? a.map_words : hash_slots_of(total, a.cap_slots, a.hash_twelfths);
  const int empty = a.map_words > 0 ? 0 : -1;
  for (int i = threadIdx.x; i < HT / 4; i += blockDim.x)
    reinterpret_cast<int4*>(table)[i] = make_int4(empty, empty, empty, empty);
  __syncthreads();
  {
    const int maxlen = kRows ? a.table_len : a.lr;
    int lps          = 1;
    while (lps < maxlen && lps < kThreads)
      lps <<= 1;
    const int within0 = threadIdx.x & (lps - 1);
    const int spp     = kThreads / lps;  // segments per pass
    const int seg0    = threadIdx.x / lps;
    // the large arrays pass through the L2 cache without staying when the sketch is to be kept there
    const bool stream = a.keep_sketch != 0 && (!kDealt || !kRows || a.table_map.ptrs == nullptr);
    const unsigned long long spol = l2_policy_stream();
    // loop bounds are the same for every thread: the slot counter below is updated once per warp
    for (int wb = 0; wb < maxlen; wb += lps) {
      const int w0 = wb + within0;
      // A wave's next four entries are on their way while four go into the set, and none is looked at for room: there
      // is a place for every entry (thousand cycles of the gathers, us a search, without either and with both: 1 000
      // queries with default parameters 327 and 321, three waves of 16 384 entries 113.5 and 108.8, 8 266 and 8 133, of
      // 32 768 ranked by sketch distance 63.0 and 56.5, 3 674 and 3 555). Lists lose: their rounds are short, and held
      // by the registers (10 000 x 1 024 entries 380 us, ahead 385, not 373).
      int ahead[4];
      auto fetch = [&](int sb) {
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const int s = sb + seg0 + u * spp;
          ahead[u]    = -1;
          if (s < nseg && w0 < maxlen) {
            if constexpr (kRows) {
              const int* at = row_of<kDealt>(a.table, a.table_map, st[s], a.table_len) + w0;
              ahead[u]      = stream ? ldg_i32_hint(at, spol) : __ldg(at);
            } else {
              const int* at = a.lists + static_cast<int64_t>(s) * a.stride + st[s] + w0;
              if (w0 < len[s]) ahead[u] = stream ? ldg_i32_hint(at, spol) : __ldg(at);
            }
          }
        }
      };
      if (kAhead) fetch(0);
      for (int sb = 0; sb < nseg; sb += 4 * spp) {
        if (!kAhead) fetch(sb);
        int v[4];
#pragma unroll
        for (int u = 0; u < 4; u++)
          v[u] = ahead[u];
        if (kAhead && sb + 4 * spp < nseg) fetch(sb + 4 * spp);
        int mine = 0;
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const int id = v[u];
          bool is_new  = false;
          if (id >= 0) {  // else nothing read, or the padding of a table row
            if (a.map_words > 0) {
              const unsigned bit = 1u << (id & 31);
              is_new             = (atomicOr(reinterpret_cast<unsigned*>(&table[id >> 5]), bit) & bit) == 0;
            } else {
              is_new = claim(table, HT, id);
            }
          }
          if (!is_new) v[u] = -1;
          mine += is_new;
        }
        // slots for the new ids of the whole warp with one update of the counter
        __syncwarp();
        int inc = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int up = __shfl_up_sync(0xffffffffu, inc, o);
          if (lane >= o) inc += up;
        }
        int base = 0;
        if (lane == 31 && inc > 0) base = atomicAdd(&ctrl[kDistinct], inc);
        base   = __shfl_sync(0xffffffffu, base, 31);
        int at = base + inc - mine;
#pragma unroll
        for (int u = 0; u < 4; u++)
          if (v[u] >= 0) {
            cand[at++] = v[u];
          }
      }
    }
  }
  __syncthreads();
  const int n = min(ctrl[kDistinct], a.nmax);
  tick(1);

  // int8 sketch distances (search_kernels.cuh:228-251), sixteen codes per lane, S / 16 lanes
  // (rounded up to a power of two) per row
  if (!int_form) {
    const float* qv = reinterpret_cast<const float*>(w16);
    if (S <= 16) {
      sketch_rows_f32<1, kDealt, kAhead>(cand, n, a.sketch, a.sketch_map, S, kq, qv, dist);
    } else if (S <= 32) {
      sketch_rows_f32<2, kDealt, kAhead>(cand, n, a.sketch, a.sketch_map, S, kq, qv, dist);
    } else if (S <= 64) {
      sketch_rows_f32<4, kDealt, kAhead>(cand, n, a.sketch, a.sketch_map, S, kq, qv, dist);
    } else if (S <= 128) {
      sketch_rows_f32<8, kDealt, kAhead>(cand, n, a.sketch, a.sketch_map, S, kq, qv, dist);
    } else if (S <= 256) {
      sketch_rows_f32<16, kDealt, kAhead>(cand, n, a.sketch, a.sketch_map, S, kq, qv, dist);
    } else {
      sketch_rows_f32<32, kDealt, kAhead>(cand, n, a.sketch, a.sketch_map, S, kq, qv, dist);
    }
  } else {
    const bool keep = a.keep_sketch != 0 && may_prefetch<kDealt>(a.sketch_map);
    if (S <= 16) {
      sketch_rows_int<1, kDealt>(cand, n, a.sketch, a.sketch_norm, a.sketch_map, S, w16, kq, dist, keep);
    } else if (S <= 32) {
      sketch_rows_int<2, kDealt>(cand, n, a.sketch, a.sketch_norm, a.sketch_map, S, w16, kq, dist, keep);
    } else if (S <= 64) {
      sketch_rows_int<4, kDealt>(cand, n, a.sketch, a.sketch_norm, a.sketch_map, S, w16, kq, dist, keep);
    } else if (S <= 128) {
      sketch_rows_int<8, kDealt>(cand, n, a.sketch, a.sketch_norm, a.sketch_map, S, w16, kq, dist, keep);
    } else if (S <= 256) {
      sketch_rows_int<16, kDealt>(cand, n, a.sketch, a.sketch_norm, a.sketch_map, S, w16, kq, dist, keep);
    } else {
      sketch_rows_int<32, kDealt>(cand, n, a.sketch, a.sketch_norm, a.sketch_map, S, w16, kq, dist, keep);
    }
  }
  __syncthreads();
  tick(2);
  if (a.tap_cand != nullptr) {
    for (int i = threadIdx.x; i < min(n, a.tap_cap); i += blockDim.x) {
      a.tap_cand[static_cast<int64_t>(q) * a.tap_cap + i] = cand[i];
      a.tap_dist[static_cast<int64_t>(q) * a.tap_cap + i] = dist[i];
    }
    if (threadIdx.x == 0) a.tap_n[q] = n;
  }

  // the nearest by (sketch distance, id) (search_kernels.cuh:259-322 takes equal distances at the
  // cut in any order)
  const int R   = a.sketch_rank ? a.KO : a.R;
  int ns        = n;
  bool selected = false;
  auto hi_at = [&](int i) { return __float_as_uint(dist[i]); };
  auto lo_at = [&](int i) { return static_cast<unsigned>(cand[i]); };
  auto emit  = [&](unsigned high, unsigned low) {
    const int s = atomicAdd(&ctrl[kEmitted], 1);
    if (s < R) {
      sid[s] = static_cast<int>(low);
      sdv[s] = __uint_as_float(high);
    }
  };
  // A search that ranks by sketch distance keeps what it selects here, so a key beyond the last one of a
  // full kept list is out already, and the others move up to the front of the candidates: a selection has only these
  // to go through, and where they fit there is none: which of them stay is the merge's to say, and the kept list
  // comes out the same. What is moved has been read by every thread, and goes no further than that. us a search, the
  // selection over all candidates and over these: 2 500 embeddings, 512 start points and three waves 3 336 and
  // 3 251, 10 000 with 128 and three 1 735 and 1 691.
  if (kRows && a.sketch_rank && ctrl[kValid] == a.KO) {
    const unsigned long long bound = rank_key(kd[a.KO - 1], static_cast<unsigned>(kid[a.KO - 1]));
    if constexpr (kShort) {
      for (int i = threadIdx.x; i < n; i += kThreads)
        if (__float_as_uint(dist[i]) <= static_cast<unsigned>(bound >> 32) &&
            rank_key(dist[i], static_cast<unsigned>(cand[i])) < bound) {
          const int s = atomicAdd(&ctrl[kWithin], 1);
          if (s < R) {
            sid[s] = cand[i];
            sdv[s] = dist[i];
          }
        }
      __syncthreads();
      selected = ctrl[kWithin] <= R;
      if (selected) ns = ctrl[kWithin];
    } else {
      for (int i0 = 0; i0 < n; i0 += 4 * kThreads) {
        float d[4];
        int id[4];
        bool within[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const int i = i0 + u * kThreads + threadIdx.x;
          d[u]        = i < n ? dist[i] : INFINITY;
          within[u]   = i < n && __float_as_uint(d[u]) <= static_cast<unsigned>(bound >> 32);
          id[u]       = within[u] ? cand[i] : 0;
          within[u]   = within[u] && rank_key(d[u], static_cast<unsigned>(id[u])) < bound;
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < 4; u++)
          if (within[u]) {
            const int s = atomicAdd(&ctrl[kWithin], 1);
            cand[s]     = id[u];
            dist[s]     = d[u];
          }
      }
      __syncthreads();
      ns       = ctrl[kWithin];
      selected = true;
      if (ns > R) {
        find_range(hi_at, ns, ctrl);
        take_smallest(hi_at, lo_at, ns, R, hist, ctrl, emit);
        ns = R;
      } else {
        for (int i = threadIdx.x; i < ns; i += blockDim.x) {
          sid[i] = cand[i];
          sdv[i] = dist[i];
        }
      }
    }
  }
  if (!selected && n > R) {
    find_range(hi_at, n, ctrl);
    take_smallest(hi_at, lo_at, n, R, hist, ctrl, emit);
    ns = R;
  } else if (!selected) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      sid[i] = cand[i];
      sdv[i] = dist[i];
    }
  }
  __syncthreads();

  tick(3);
  // The set of kept ids, where the set of the gather was. In a region of its own it is made with the start
  // points and saves these two barriers, which brings nothing (300 queries of 20 000 rows 82.4 and 81.6 us a
  // search, 10 000 of a million 869 and 866, apart and here), but can cost blocks: 512 start points x 32 entries 1 174
  // and 1 032, 128 x 16 with 512 reranked rows of 512 bytes 2 177 and 2 022.
  if constexpr (kRows) {
    for (int i = threadIdx.x; i < a.kept_slots; i += kThreads)
      table[i] = -1;
    __syncthreads();
    for (int i = threadIdx.x; i < a.KO; i += kThreads)
      insert_id(table, a.kept_slots, kid[i]);
    __syncthreads();
  }
  // A selected id that is already in the kept list brings the key it already has there: drop it
  // before the vectors are read (the reference reranks it again and collapses the equal keys). Every row
  // about to be read is asked for at once (128-byte lines into L2), so the distance loop below finds
  // most of them on the way; not wide rows, of which the loop has enough on the way itself. us a search, asked for and
  // not, 1 000 queries at 128 rows a round, at 512, and 5 000 at 128 and 384: 512 bytes a row 421 and 425, 723 and 722, 681 and
  // 682; 768 bytes 421 and 425, 737 and 728, 766 and 753; 1 024 bytes 426 and 432, 759 and 743, 876 and 853; 1 920 bytes 500 and
  // 502, 992 and 944, 1 360 and 1 265. (64 wide rows a round are the exception, 1 024 bytes 333 and 339, 1 920 393 and 402.)
  const int row_bytes = a.D * 2;
  const bool ahead    = !a.sketch_rank && row_bytes <= kAheadBytes && may_prefetch<kDealt>(a.vector_map);
  for (int r = threadIdx.x; r < ns; r += blockDim.x) {
    const int v = sid[r];
    if (kRows && holds_id(table, a.kept_slots, v)) {
      sid[r] = -1;
    } else if (ahead) {
      const char* row = reinterpret_cast<const char*>(a.vectors + static_cast<int64_t>(v) * a.D);
      for (int b = 0; b < row_bytes; b += 128)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(row + b));
    }
  }
  if (kRows) __syncthreads();
  int reranked = 0;
  if (!a.sketch_rank) {
    if (a.stats != nullptr) {
      int mine = 0;
      for (int i = threadIdx.x; i < ns; i += blockDim.x)
        mine += sid[i] >= 0;
      block_scan<kThreads>(mine, wsum, reranked);
    }
    tick(4);
    // (rows of other GPUs do not pass through this cache)
    if (!kDealt && a.pass_vectors != 0)
      exact_distances<kDealt, true>(sid, ns, a.vectors, a.vector_map, a.D, fq, sdv);
    else
      exact_distances<kDealt, false>(sid, ns, a.vectors, a.vector_map, a.D, fq, sdv);
    tick(5);
  }
  merge_into_kept(pool, sorted, a.P, pb, pd, a.KO, kid, kd, kRows ? ctrl[kValid] : 0, sid, sdv, ns, hist, ctrl,
                  a.out_i == nullptr ? nullptr : a.out_i + static_cast<int64_t>(q) * a.k,
                  a.out_i == nullptr ? nullptr : a.out_d + static_cast<int64_t>(q) * a.k,
                  a.out_i == nullptr ? 0 : a.k);
  tick(6);
  if (a.stats != nullptr && threadIdx.x == 0) {
    long long* s = a.stats + static_cast<int64_t>(q) * 8;
    if constexpr (kRows) {
      s[4] += ctrl[kStarts];
      s[5] += n;
    } else {
      s[2] += total;
      s[3] += n;
    }
    if (!a.sketch_rank) s[6] += ns;  // rows the reference reranks
    s[7] += reranked;  // rows read here (those already kept are skipped)
  }
}

// search_kernels.cuh:634-669: exact distances of the first R kept entries, best k of them.
__global__ void __launch_bounds__(kRoundThreads) final_rerank_kernel(const long long* __restrict__ si,
                                                                     int KO,
                                                                     int R,
                                                                     const __half* __restrict__ vectors,
                                                                     const row_map vector_map,
                                                                     int D,
                                                                     const float* __restrict__ Q,
                                                                     int k,
                                                                     int P,
                                                                     long long* __restrict__ bi,
                                                                     float* __restrict__ bd,
                                                                     long long* __restrict__ stats)
{
  extern __shared__ __align__(16) int smem[];
  unsigned long long* pool   = reinterpret_cast<unsigned long long*>(smem);  // [k + R]
  unsigned long long* sorted = pool + ((k + R + 1) & ~1);                    // [P]
  int* sid                   = reinterpret_cast<int*>(sorted + max(2 * P, 64));  // sorted [max(2 P, 64)]; sid [R]
  float* sdv                 = reinterpret_cast<float*>(sid + ((R + 3) & ~3));
  float* fq                  = sdv + ((R + 3) & ~3);                         // [D]
  unsigned* hist             = reinterpret_cast<unsigned*>(fq + ((D + 63) & ~63));
  int* wsum                  = reinterpret_cast<int*>(hist + 256);
  int* ctrl                  = wsum + 32;
  const int q                = blockIdx.x;
  const long long* ps        = si + static_cast<int64_t>(q) * KO;
  if (threadIdx.x == 0) ctrl[kMerged] = 0;
  wait_for_previous_kernel();
  for (int i = threadIdx.x; i < D; i += blockDim.x)
    fq[(D & 7) ? i : query_slot(i)] = Q[static_cast<int64_t>(q) * D + i];
  // the kept list is packed (valid entries first), so the valid ones among the first R are a prefix
  int mine = 0;
  for (int i = threadIdx.x; i < R; i += blockDim.x) {
    const long long v = ps[i];
    sid[i]            = static_cast<int>(v);
    if (v >= 0) mine++;
  }
  int ns = 0;
  block_scan(mine, wsum, ns);
  exact_distances<true, false>(sid, ns, vectors, vector_map, D, fq, sdv);
  merge_into_kept(pool, sorted, P, bi + static_cast<int64_t>(q) * k, bd + static_cast<int64_t>(q) * k,
                  k, nullptr, nullptr, 0, sid, sdv, ns, hist, ctrl);
  if (stats != nullptr && threadIdx.x == 0) {
    stats[static_cast<int64_t>(q) * 8 + 6] += ns;
    stats[static_cast<int64_t>(q) * 8 + 7] += ns;
  }
}

// search_kernels.cuh:517-564: kept lists of nsrc sources -> the nearest copy of each id -> best
// KO. The sources are rows of arrays in this GPU's own memory (the exchange brought them here).
__global__ void merge_kept_kernel(const long long* __restrict__ src_i,
                                  const float* __restrict__ src_d,
                                  int nsrc,
                                  int64_t src_stride,
                                  int KO,
                                  int P,
                                  long long* __restrict__ si,
                                  float* __restrict__ sd)
{
  extern __shared__ __align__(16) int smem[];
  unsigned long long* mk = reinterpret_cast<unsigned long long*>(smem);
  const int q            = blockIdx.x;
  const int total        = nsrc * KO;
  for (int i = threadIdx.x; i < P; i += blockDim.x) {
    unsigned long long k = kNoKey;
    if (i < total) {
      const int h       = i / KO;
      const int64_t at  = h * src_stride + static_cast<int64_t>(q) * KO + i % KO;
      const long long v = src_i[at];
      if (v >= 0)
        k = (static_cast<unsigned long long>(static_cast<unsigned>(v)) << 32) | __float_as_uint(src_d[at]);
    }
    mk[i] = k;
  }
  __syncthreads();
  bitonic_sort(mk, P);  // by (id, distance): the first key of an id run is its nearest copy
  const int per = (P + kRoundThreads - 1) / kRoundThreads;
  const int i0  = threadIdx.x * per;
  unsigned long long mine[4096 / kRoundThreads];
  int cnt = 0;
  for (int i = i0; i < min(P, i0 + per); i++) {
    const unsigned long long k = mk[i];
    unsigned long long out     = kNoKey;
    if (k != kNoKey && (i == 0 || (mk[i - 1] >> 32) != (k >> 32)))
      out = ((k & 0xffffffffULL) << 32) | (k >> 32);
    mine[cnt++] = out;
  }
  __syncthreads();
  cnt = 0;
  for (int i = i0; i < min(P, i0 + per); i++)
    mk[i] = mine[cnt++];
  __syncthreads();
  bitonic_sort(mk, P);  // by (distance, id)
  long long* pb = si + static_cast<int64_t>(q) * KO;
  float* pd     = sd + static_cast<int64_t>(q) * KO;
  for (int i = threadIdx.x; i < KO; i += blockDim.x) {
    const unsigned long long k = mk[i];
    pb[i] = k == kNoKey ? -1 : static_cast<long long>(static_cast<unsigned>(k & 0xffffffffULL));
    pd[i] = k == kNoKey ? INFINITY : __uint_as_float(static_cast<unsigned>(k >> 32));
  }
}

}  // namespace

size_t round_smem_bytes(const round_args& a) { return sizeof(int) * round_layout(a).words; }

/// Threads per query block. A multiprocessor runs 1024 threads of this kernel whatever the block size
/// (64 registers each): a.threads makes the most of the blocks its shared memory holds. A batch of
/// fewer blocks than the multiprocessors can hold at once is a matter of latency: its blocks get as
/// many threads as still run side by side. us a search, with that and with a.threads: 1 query of 64 copies
/// 64 and 81, 300 queries 91 and 105, 592 100 and 107, from 800 on the same; 100 queries with 256 start
/// points 180 and 226. Rounds of a few hundred entries lose to the wider barriers (one query of 8 copies x
/// 8 entries: 59 and 54).
int round_threads(const round_args& a)
{
  int threads = a.threads;
  while (threads < 1024 && static_cast<int64_t>(a.m) * threads * 2 <= int64_t{1024} * a.sms)
    threads *= 2;
  return threads;
}

namespace {

/// Whether this is a short wave (round_kernel), of those that take blocks of 1 024 threads only because there are few
/// queries. us a search with the longer code and with the shorter, 64 neighbors a start point, 1, 8 and 60 queries: 16 start
/// points and three waves 94.1 and 92.6, 95.2 and 94.4, 103.5 and 103.1; 64 114.4 and 113.6, 122.3 and 122.6, 134.0 and
/// 134.4; 128 and two 114.0 and 113.9 (descriptors 87.2 and 86.6), 123.2 and 124.3, 137.9 and 137.1; 256 123.9 and 124.4, 139.0 and
/// 140.4, 157.0 and 156.4. Ranked by sketch distance 32 and two, 1 and 30 queries 80.8 and 80.3, 86.9 and 87.6; 128 111.4
/// and 113.6.
bool short_wave(const round_args& a)
{
  return a.threads < 1024 && a.nmax <= (a.sketch_rank ? 2048 : 8192) && static_cast<int64_t>(a.m) * a.nmax <= 16384;
}

/// Launch that may begin while the kernel before it in the stream is finishing; the kernel waits for
/// it where it first needs its results (wait_for_previous_kernel).
/// Only where it matters, in batches that leave multiprocessors idle: us a search of one round and one
/// wave, early and not, 1 query 64 and 72, 100 queries 82 and 86, 148 84 and 86, 800 124 and 115, 1 000 132
/// and 126, 10 000 617 and 620. (The first blocks of a kernel that starts under the last of another find the
/// L1 cache split for the other's shared memory.)
template <typename... P, typename... A>
void launch_overlapped(bool early, void (*kernel)(P...), unsigned grid, unsigned threads, size_t smem, cudaStream_t s,
                       A&&... args)
{
  cudaLaunchConfig_t cfg{};
  cfg.gridDim          = dim3(grid);
  cfg.blockDim         = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream           = s;
  cudaLaunchAttribute at{};
  at.id                                         = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = early ? 1 : 0;
  cfg.attrs                                     = &at;
  cfg.numAttrs                                  = 1;
  cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

template <bool kRows, bool kDealt, int kThreads, bool kShort = false>
void launch_round(const round_args& a, cudaStream_t s)
{
  launch_overlapped(a.m <= a.sms, round_kernel<kRows, kDealt, kThreads, kShort>, static_cast<unsigned>(a.m), kThreads, round_smem_bytes(a), s, a);
}
template <bool kRows, bool kDealt>
void launch_round(const round_args& a, cudaStream_t s)
{
  switch (round_threads(a)) {
    case 1024:
      if (kRows && short_wave(a))
        launch_round<kRows, kDealt, 1024, kRows>(a, s);
      else
        launch_round<kRows, kDealt, 1024>(a, s);
      break;
    case 512: launch_round<kRows, kDealt, 512>(a, s); break;
    case 256: launch_round<kRows, kDealt, 256>(a, s); break;
    default: launch_round<kRows, kDealt, 128>(a, s); break;
  }
}
template <bool kRows, bool kDealt>
void allow_smem()
{
  cudaFuncSetAttribute(round_kernel<kRows, kDealt, 128, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxBlockSmem);
  cudaFuncSetAttribute(round_kernel<kRows, kDealt, 256, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxBlockSmem);
  cudaFuncSetAttribute(round_kernel<kRows, kDealt, 512, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxBlockSmem);
  cudaFuncSetAttribute(round_kernel<kRows, kDealt, 1024, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxBlockSmem);
  cudaFuncSetAttribute(round_kernel<kRows, kDealt, 1024, kRows>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxBlockSmem);
}
bool dealt(const round_args& a)
{
  return a.table_map.ptrs != nullptr || a.sketch_map.ptrs != nullptr || a.vector_map.ptrs != nullptr;
}
}  // namespace

void round_allow_smem()
{
  allow_smem<false, false>();
  allow_smem<true, false>();
  allow_smem<false, true>();
  allow_smem<true, true>();
}

void round_lists(const round_args& a, cudaStream_t s)
{
  if (a.m <= 0) return;
  if (dealt(a))
    launch_round<false, true>(a, s);
  else
    launch_round<false, false>(a, s);
}

void round_rows(const round_args& a, cudaStream_t s)
{
  if (a.m <= 0) return;
  if (dealt(a))
    launch_round<true, true>(a, s);
  else
    launch_round<true, false>(a, s);
}

void final_rerank(const long long* si, int KO, int R, const __half* vectors, row_map vector_map, int D,
                  const float* Q, int k, int m, long long* bi, float* bd, long long* stats,
                  cudaStream_t s)
{
  if (m <= 0) return;
  int P = 2;
  while (P < k)
    P <<= 1;
  const size_t words = 2 * static_cast<size_t>((k + R + 1) & ~1) + 2 * static_cast<size_t>(std::max(2 * P, 64)) +
                       2 * static_cast<size_t>((R + 3) & ~3) + ((D + 63) & ~63) + 256 + 32 + kCtlWords;
  // early while there is a multiprocessor for every block, as in launch_round
  launch_overlapped(m <= 128, final_rerank_kernel, static_cast<unsigned>(m), kRoundThreads, sizeof(int) * words, s, si, KO, R,
                    vectors, vector_map, D, Q, k, P, bi, bd, stats);
}

void merge_kept(const long long* src_i, const float* src_d, int nsrc, int64_t src_stride, int KO,
                int P, int m, long long* si, float* sd, cudaStream_t s)
{
  if (m <= 0) return;
  const size_t smem = sizeof(int) * (2 * static_cast<size_t>(P) + 16);
  if (smem > (48 << 10))  // per device and context, so asked for whenever it is needed
    cudaFuncSetAttribute(merge_kept_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 8 * 4096 + 64);
  merge_kept_kernel<<<m, kRoundThreads, smem, s>>>(src_i, src_d, nsrc, src_stride, KO, P, si, sd);
}

}  // namespace octex_b200::kernels
