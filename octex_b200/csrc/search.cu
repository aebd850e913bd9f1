// Batched search: plan (limits, buffers, the graph of a batch that stays in them) and the per-batch loop.
//
// Answers cpp/src/neighbors/octex/search.cu of hpdic/octex (make_plan :619-794, get_plan :796-814,
// search_impl :816-961, the two search overloads :1020-1064) for one process per GPU. Parameter
// limits and error texts are the reference's. A batch is two kernels and one per wave: projection
// with cell lookup and sketch-space queries, first round, waves, the last of which writes the
// results. Queries and results in the memory of the index's GPU are used where they are, on the caller's
// stream (the batches of a call of several on a second one in turn, the second half of a large batch on
// another), and every kernel is launched for the queries there are: no copies, no padding. A batch that
// stays in the plan's buffers (resident searches, several processes) is replayed as one CUDA graph.

#include "search_impl.hpp"

#include <algorithm>
#include <array>
#include <cmath>
#include <cstring>

namespace octex_b200 {

namespace detail {

namespace {

constexpr size_t kPiece = 256;  // arrays of a plan begin on such boundaries

/// The rest of the plan's memory is to hold arrays of these sizes.
void reserve(plan& pl, int device, std::initializer_list<size_t> bytes)
{
  size_t total = 0;
  for (size_t b : bytes)
    total += (b + kPiece - 1) / kPiece * kPiece;
  pl.memory.emplace_back(device, total);
  pl.memory_used = 0;
}

/// An array of the plan: a piece of the memory reserved for it, where there is room, else of a new block.
template <typename T>
auto alloc(plan& pl, int device, int64_t count, int fill = -2) -> dbuf
{
  const size_t bytes = static_cast<size_t>(std::max<int64_t>(count, 1)) * sizeof(T);
  if (pl.memory.empty() || pl.memory.back().size - pl.memory_used < bytes) reserve(pl, device, {bytes});
  const dbuf b = dbuf::borrow(device, pl.memory.back().as<char>() + pl.memory_used, bytes);
  pl.memory_used += std::min((bytes + kPiece - 1) / kPiece * kPiece, pl.memory.back().size - pl.memory_used);
  if (fill != -2) OCTEX_CUDA_TRY(cudaMemset(b.ptr, fill, b.size));
  pl.buffer_bytes += static_cast<int64_t>(bytes);
  return dbuf::borrow(device, b.ptr, bytes);
}

/// The kernels' view of an array dealt by rows (empty when the array is whole).
auto map_of(index_impl const& ix, dealt_rows const& d) -> kernels::row_map
{
  kernels::row_map m;
  if (!d.on) return m;
  OCTEX_EXPECTS(d.ptrs.ptr != nullptr,
                "octex: the index holds row ranges of other processes: connect the processes first "
                "(octexB200CommInit)");
  OCTEX_EXPECTS(d.rows_per < (int64_t{1} << 31), "octex: more than 2^31 rows per process");
  m.ptrs  = d.ptrs.as<long long>();
  m.rows  = static_cast<int>(d.rows_per);
  m.local = static_cast<int>(std::min<int64_t>(d.row0, ix.n - 1));
  return m;
}

constexpr size_t kSmemSoftLimit = size_t{96} << 10;   // above this the candidates go to global memory
constexpr size_t kSmemHardLimit = kernels::kMaxBlockSmem;
// a block above this (1 KB is the system's) gets the whole 228 KB step of a multiprocessor's 256 KB, which
// leaves the L1 cache 28 KB instead of 60
constexpr size_t kSmemBelowLastStep = (size_t{196} << 10) - 1024;

/// Blocks of a multiprocessor, by shared memory (1 KB per block is the system's).
auto blocks_of(kernels::round_args const& r) -> size_t { return (size_t{228} << 10) / (kernels::round_smem_bytes(r) + 1024); }

/// Fill the size fields of a round and decide where its candidate arrays live.
void size_round(plan& pl, kernels::round_args& r, int entries_max, bool waves, int pick_entries, int device,
                int64_t sketch_bytes, int64_t rows, bool vectors_here)
{
  r.pick_slots = 0;
  if (pick_entries > 0) {
    r.pick_slots = 64;
    while (r.pick_slots * 3 < pick_entries * 4)  // at most 75 % full
      r.pick_slots <<= 1;
  }
  r.kept_slots = 0;  // the set of kept ids a wave filters its selection with
  if (waves) {
    r.kept_slots = 64;
    while (r.kept_slots < 2 * r.KO)
      r.kept_slots <<= 1;
  }
  r.nmax = std::max(entries_max, 1);
  r.P    = 2;
  while (r.P < r.KO)
    r.P <<= 1;
  r.cand_global = nullptr;
  r.dist_global = nullptr;
  // the gather's hash set: half full at most when eight blocks still fit a multiprocessor's shared
  // memory (1 KB per block is the system's), else two thirds, else three quarters
  constexpr size_t kEightBlocks = (size_t{228} << 10) / 8 - 1024;
  for (int twelfths : {24, 18, 16}) {
    r.hash_twelfths = twelfths;
    r.cap_slots = kernels::hash_slots_of(std::min(entries_max, kernels::kMaxHash), kernels::kMaxHash, twelfths);
    r.ht_slots  = std::max({r.cap_slots, r.pick_slots, r.kept_slots});
    if (kernels::round_smem_bytes(r) <= kEightBlocks) break;
  }
  // placeholders: non-null makes the layout drop the two arrays; the real buffers follow
  auto settle = [&] {
    r.cand_global = nullptr;
    r.dist_global = nullptr;
    if (kernels::round_smem_bytes(r) > kSmemSoftLimit) {
      r.cand_global = reinterpret_cast<int*>(1);
      r.dist_global = reinterpret_cast<float*>(1);
    }
    return blocks_of(r);
  };
  // A bit for every row of the index instead of the set, where that takes no more room, or where the set
  // leaves a multiprocessor one block anyway: one exchange an entry, and no way to a free slot.
  // us a search, two waves by the set and by bits where these take no more room: 100 003 rows, 8 192 entries 502 and
  // 487; a million, 32 768 entries ranked by sketch distance, three waves 4 340 and 3 798. One block either way and more
  // room (19 200 entries; 22 400): a million rows 1 708 and 1 587; 1 695 and 1 575; 1.4 million 1 757 and 1 640. With the
  // last step of shared memory the bits lose: 32 768 entries, 1.4 million rows 1 771 and 1 869, 1.5 million 1 791 and
  // 1 903 (ranked by sketch distance 4 019 and 3 927, 4 065 and 4 035). Where two blocks fit with the set the bits at one
  // lose what the blocks do side by side: a million rows, 16 384 entries, three waves 8 670 and 9 605.
  const size_t blocks = settle();
  const int slots     = r.ht_slots;
  const int words     = static_cast<int>(std::min<int64_t>((rows + 127) / 128 * 4, 1 << 20));
  if (words <= slots || blocks < 2) {
    r.map_words = words;
    r.ht_slots  = std::max({words, r.pick_slots, r.kept_slots, slots >= r.nmax ? r.nmax : 0});
    settle();
    if (r.ht_slots > slots && kernels::round_smem_bytes(r) > kSmemBelowLastStep) {
      r.map_words = 0;
      r.ht_slots  = slots;
      settle();
    }
  }
  OCTEX_EXPECTS(kernels::round_smem_bytes(r) <= kSmemHardLimit, "octex: the round does not fit shared memory");
  if (r.cand_global != nullptr) {
    pl.scratch_cand.push_back(alloc<int>(pl, device, int64_t{r.m} * r.nmax));
    r.cand_global = pl.scratch_cand.back().as<int>();
    // the sketch distances still go where the hash set was when that region holds them all (the
    // selection makes several passes over them)
    r.dist_global = nullptr;
    if (r.ht_slots < r.nmax) {
      pl.scratch_dist.push_back(alloc<float>(pl, device, int64_t{r.m} * r.nmax));
      r.dist_global = pl.scratch_dist.back().as<float>();
    }
  }
  // threads per block: a multiprocessor runs 1024 threads of this kernel (64 registers each); when
  // fewer than eight blocks fit its shared memory, the blocks get more threads to make up for it
  const size_t held = blocks_of(r);
  r.threads         = held >= 8 ? 128 : held >= 4 ? 256 : held >= 2 ? 512 : 1024;
  OCTEX_CUDA_TRY(cudaDeviceGetAttribute(&r.sms, cudaDevAttrMultiProcessorCount, device));
  {
    // the sketch stays in the L2 cache when it and its constants take at most 60 % of it
    int l2 = 0;
    OCTEX_CUDA_TRY(cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, device));
    r.keep_sketch = sketch_bytes > 0 && static_cast<double>(sketch_bytes) <= 0.6 * l2 ? 1 : 0;
    // One that takes a quarter of it or more is pushed out in part by the fp16 rows, read once or twice a batch,
    // unless those go first. us a search with the rows as others and first, 10 000 queries at 384 rows a wave and
    // 2 000 at 512 and three waves: 68 MB of sketch 1 093 and 1 075, 1 896 and 1 839; 36 MB 924 and 920, 1 328 and 1 289; 34 MB
    // 1 016 and 1 020, 1 446 and 1 434. A smaller sketch stays anyway, and rows that many queries share are better
    // kept: 31 MB 1 036 and 1 045, 1 445 and 1 436; 27 MB 1 001 and 1 008, 1 405 and 1 397; 13 MB, rows of 1 920 bytes
    // 2 184 and 2 308, 1 156 and 1 180. (Rows that wide lose above the line too where the data has few clusters, and with
    // default parameters win: 53 MB 2 612 and 2 648, 2 001 and 2 025, 513 and 497.) Rows in host memory come over the
    // bus and are kept at any size: 2 000 queries of 400 000 x 96 4 682 and 4 957.
    r.pass_vectors = vectors_here && r.keep_sketch != 0 && static_cast<double>(sketch_bytes) >= 0.25 * l2 ? 1 : 0;
  }
}

}  // namespace

plan::~plan()
{
  int cur = 0;
  cudaGetDevice(&cur);
  cudaSetDevice(device);
  if (used) cudaEventSynchronize(done_ev);  // its kernels may be running on a caller's stream
  if (graph != nullptr) cudaGraphExecDestroy(graph);
  if (done_ev != nullptr) cudaEventDestroy(done_ev);
  if (join_ev != nullptr) cudaEventDestroy(join_ev);
  memory.clear();  // the release waits for what still runs, replays of a caller's capture too
  if (words != nullptr) words->give_back(word);
  cudaSetDevice(cur);
}

/// A wait inside the tensor-core projection gave up (it never does unless the GPU misbehaves):
/// report it once and clear the word, so that one event does not poison the calls after it. Call
/// it when the stream of the plan is idle.
void check_tc(plan const& pl)
{
  if (pl.tc_error_host == nullptr || *pl.tc_error_host == 0) return;
  const int code    = *pl.tc_error_host;
  *pl.tc_error_host = 0;
  throw error("octex: the projection gave up waiting for data it had asked for (code " + std::to_string(code) +
              "); the results of that batch are not valid");
}

auto round_shapes(plan const& pl) -> std::vector<int32_t>
{
  std::vector<int32_t> out;
  for (auto const* r : {&pl.r1, &pl.r2}) {
    const bool any = r == &pl.r1 || pl.sp.waves > 0;
    const auto put = [&](int64_t v) { out.push_back(any ? static_cast<int32_t>(v) : 0); };
    put(any ? kernels::round_threads(*r) : 0);
    put(any ? blocks_of(*r) : 0);
    put(r->map_words > 0 ? 0 : r->cap_slots);
    put(r->map_words);
    put(r->cand_global != nullptr);
    put(r->pass_vectors);
  }
  return out;
}

auto batch_forms(plan const& pl) -> std::vector<int32_t>
{
  return {static_cast<int32_t>(pl.halves_from), pl.halved ? 1 : 0, static_cast<int32_t>(pl.projected.form), pl.projected.rows};
}

/// Where a batch's queries are and its results go (device-accessible memory).
struct batch_io {
  const float* q;
  long long* ids;
  float* dist;
};

/// The plan's own buffers.
auto own_io(plan const& pl) -> batch_io { return {pl.qbuf.as<float>(), pl.bi, pl.bd}; }

auto capturing(cudaStream_t s) -> bool
{
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  OCTEX_CUDA_TRY(cudaStreamIsCapturing(s, &cap));
  return cap != cudaStreamCaptureStatusNone;
}

/// What is queued on s from here on comes after the plan's last batch, whose buffers it uses.
void follow_last_batch(plan& pl, cudaStream_t s)
{
  // a graph the caller is capturing is ordered by whoever launches it (and a capturing stream does not
  // say its id)
  if (!pl.used || capturing(s)) return;
  unsigned long long id = 0;
  OCTEX_CUDA_TRY(cudaStreamGetId(s, &id));
  if (id != pl.last_stream) OCTEX_CUDA_TRY(cudaStreamWaitEvent(s, pl.done_ev, 0));
}

/// The plan's last batch is what s holds now.
void mark_last_batch(plan& pl, cudaStream_t s)
{
  if (capturing(s)) return;
  OCTEX_CUDA_TRY(cudaEventRecord(pl.done_ev, s));
  OCTEX_CUDA_TRY(cudaStreamGetId(s, &pl.last_stream));
  pl.used = true;
}

/// Rows of a batch by one process.
struct row_range {
  int first, count;
};

/// Launch every kernel of a batch of pl.m queries on s (captured into the graph, or run directly), or (part given:
/// by one process and without observation) of some of its rows. io is the whole batch's.
void run_batch(index_impl const& ix, plan& pl, batch_io const& io, cudaStream_t s, std::vector<cudaEvent_t>* marks,
               row_range const* part = nullptr)
{
  const int64_t first = part != nullptr ? part->first : 0;
  const int m1 = part != nullptr ? part->count : pl.m1, mw = part != nullptr ? part->count : pl.mw;
  pl.halved    = part != nullptr;
  pl.projected = {};
  // marks (profiling only): one event before the first kernel and one after every step
  auto mark = [&] {
    if (marks == nullptr) return;
    cudaEvent_t e = nullptr;
    OCTEX_CUDA_TRY(cudaEventCreate(&e));
    OCTEX_CUDA_TRY(cudaEventRecord(e, s));
    marks->push_back(e);
  };
  auto const& p  = ix.part;
  const int D    = static_cast<int>(ix.dim);
  const int sw   = ix.sketch_width;
  const int L    = static_cast<int>(ix.spacings.size());
  const int wdt  = 8 * ix.blocks * p.copies;
  if (pl.stats.ptr != nullptr) {
    OCTEX_CUDA_TRY(cudaMemsetAsync(pl.stats.ptr, 0, pl.stats.size, s));
    OCTEX_CUDA_TRY(cudaMemsetAsync(pl.phase1.ptr, 0, pl.phase1.size, s));
    OCTEX_CUDA_TRY(cudaMemsetAsync(pl.phase2.ptr, 0, pl.phase2.size, s));
  }
  mark();
  float finest   = ix.spacings[0];
  for (float f : ix.spacings)
    finest = std::min(finest, f);
  kernels::sketch_job job;
  job.q = io.q + first * D, job.mean = p.mean.as<float>(), job.basis = p.basis.as<float>();
  job.m = m1, job.D = D, job.S = sw;
  job.beside = part != nullptr ? 2 : 1;
  job.qs   = pl.qs.as<float>() + first * sw;
  job.keep = io.q == pl.qbuf.as<float>() ? nullptr : pl.qbuf.as<float>() + first * D;
  kernels::tc_lookup look;
  look.table    = p.cell_table.as<kernels::cell_slot>();
  look.keys     = p.cell_keys.as<long long>();
  look.levels   = p.cell_levels.as<kernels::cell_level>();
  look.list_len = ix.list_len;
  look.lr       = pl.lr;
  look.seg      = pl.seg.as<int2>() + first * p.copies;
  look.stats    = pl.stats.as<long long>();
  // without inspection the cells are looked up where their codes are computed: no codes array, no
  // lookup kernel
  if (!pl.dbg.taps && pl.use_tc) {
    mark();
    pl.projected = kernels::project_decode_tc(pl.tc, job, L, p.shift.as<__half>(), p.inv_f.as<float>(), finest, nullptr,
                                              nullptr, look, pl.tc_error_dev, s);
    mark();
    mark();
  } else if (!pl.dbg.taps) {
    mark();
    pl.projected = kernels::project_lookup_ordered(job, ix.blocks, p.ut.as<__half>(), p.ldu, p.copies, L,
                                                   p.shift.as<__half>(), p.inv_f.as<float>(), finest, look, pl.r1.sms, s);
    mark();
    mark();
  } else {
    // everything is written out: codes of every level, coordinates, then the lookup on its own
    if (job.keep != nullptr)
      OCTEX_CUDA_TRY(cudaMemcpyAsync(job.keep, io.q, sizeof(float) * pl.m1 * D, cudaMemcpyDefault, s));
    if (pl.use_tc) {
      mark();
      job.keep = nullptr;
      kernels::project_decode_tc(pl.tc, job, L, p.shift.as<__half>(), p.inv_f.as<float>(), finest,
                                 pl.codes.as<long long>(), pl.Y.as<__half>(), kernels::tc_lookup{}, pl.tc_error_dev, s);
      mark();
    } else {
      kernels::center_sketch(pl.qbuf.as<float>(), job.mean, job.basis, pl.m1, D, sw, pl.qh.as<__half>(), p.ldu, job.qs, s);
      mark();
      kernels::project_ordered(pl.qh.as<__half>(), p.ldu, p.ut.as<__half>(), p.ldu, p.shift.as<__half>(), pl.m1, wdt, D,
                               pl.Y.as<__half>(), s);
      mark();
      kernels::decode_codes(pl.Y.as<__half>(), int64_t{pl.m1} * p.copies, ix.blocks, L, p.inv_f.as<float>(),
                            pl.codes.as<long long>(), s);
    }
    mark();
    kernels::probe(pl.codes.as<long long>(), pl.m1, p.copies, L, look, s);
  }
  mark();
  // the last round writes the results unless a kernel of its own makes them
  const bool reranks_at_end = pl.sp.sketch_rank && pl.FR > 0;
  const bool last_is_lists  = pl.sp.waves == 0 && !pl.shard;
  auto with_results         = [&](kernels::round_args r, bool last) {
    if (last && !reranks_at_end) {
      r.out_i = io.ids + first * pl.k;
      r.out_d = io.dist + first * pl.k;
      r.k     = pl.k;
    }
    if (part != nullptr) {
      r.m = part->count;
      if (r.seg != nullptr) r.seg += first * p.copies;
      r.qs += first * sw;
      r.Q += first * D;
      r.si += first * pl.KO;
      r.sd += first * pl.KO;
      if (r.done != nullptr) r.done += first * r.done_stride;
      if (r.cand_global != nullptr) r.cand_global += first * r.nmax;
      if (r.dist_global != nullptr) r.dist_global += first * r.nmax;
    }
    return r;
  };
  pl.r1.m = pl.m1;
  pl.r2.m = pl.mw;
  kernels::round_lists(with_results(pl.r1, last_is_lists), s);
  mark();
  if (pl.shard) {
    // Every process ran the first round of all m rows over its own copies. Row block [lo_r, hi_r)
    // of each kept list goes to process r (search_kernels.cuh:517-539 reads the same blocks through
    // peer pointers); then the nearest copy of every id, best KO (merge_kept_kernel).
    auto& c        = *ix.comm;
    const size_t e = static_cast<size_t>(pl.KO);
    c.group_start();
    for (int r = 0; r < pl.world; r++) {
      const int lo_r = static_cast<int>(int64_t{pl.m} * r / pl.world);
      const int hi_r = static_cast<int>(int64_t{pl.m} * (r + 1) / pl.world);
      long long* ri  = pl.recv_i.as<long long>() + static_cast<size_t>(r) * pl.mwmax * e;
      float* rd      = pl.recv_d.as<float>() + static_cast<size_t>(r) * pl.mwmax * e;
      if (r == pl.rank) {
        OCTEX_CUDA_TRY(cudaMemcpyAsync(ri, pl.si.as<long long>() + pl.lo * e, pl.mw * e * sizeof(long long),
                                       cudaMemcpyDeviceToDevice, s));
        OCTEX_CUDA_TRY(cudaMemcpyAsync(rd, pl.sd.as<float>() + pl.lo * e, pl.mw * e * sizeof(float),
                                       cudaMemcpyDeviceToDevice, s));
        continue;
      }
      c.send(pl.si.as<long long>() + lo_r * e, (hi_r - lo_r) * e * sizeof(long long), r, s);
      c.send(pl.sd.as<float>() + lo_r * e, (hi_r - lo_r) * e * sizeof(float), r, s);
      c.recv(ri, pl.mw * e * sizeof(long long), r, s);
      c.recv(rd, pl.mw * e * sizeof(float), r, s);
    }
    c.group_end();
    mark();
    kernels::merge_kept(pl.recv_i.as<long long>(), pl.recv_d.as<float>(), pl.world,
                        int64_t{pl.mwmax} * pl.KO, pl.KO, pl.P_merge, pl.mw, pl.wsi, pl.wsd, s);
    mark();
  }
  if (pl.dbg.taps && pl.mw > 0) {
    OCTEX_CUDA_TRY(cudaMemcpyAsync(pl.kept1_i.ptr, pl.wsi, sizeof(long long) * pl.mw * pl.KO,
                                   cudaMemcpyDeviceToDevice, s));
    OCTEX_CUDA_TRY(cudaMemcpyAsync(pl.kept1_d.ptr, pl.wsd, sizeof(float) * pl.mw * pl.KO,
                                   cudaMemcpyDeviceToDevice, s));
  }
  const float* Qw = pl.qbuf.as<float>() + static_cast<size_t>(pl.lo - pl.q1) * D;
  for (int wv = 0; wv < pl.sp.waves; wv++) {
    kernels::round_args r = with_results(pl.r2, wv == pl.sp.waves - 1);
    r.done_off            = wv * pl.sp.starts;
    kernels::round_rows(r, s);
    mark();
  }
  if (reranks_at_end)
    kernels::final_rerank(pl.wsi + first * pl.KO, pl.KO, pl.FR, p.vectors.as<__half>(), pl.r1.vector_map, D, Qw + first * D,
                          pl.k, mw, io.ids + first * pl.k, io.dist + first * pl.k, pl.stats.as<long long>(), s);
  else if (pl.sp.waves == 0 && pl.shard)
    kernels::take_k(pl.wsi, pl.wsd, pl.KO, pl.k, pl.mw, io.ids, io.dist, s);
  mark();
  if (pl.world > 1) {
    // every process gets the results of all slices (blocks of mwmax rows, the last rows of a
    // block unused when the slices differ in size)
    ix.comm->all_gather(pl.out.ptr, pl.gathered.ptr, pl.out_block, s);
    mark();
  }
  OCTEX_CUDA_TRY(cudaPeekAtLastError());
}

/// The slices of a batch of m queries (search.cu:666-676 of the reference).
void set_rows(plan& pl, int m)
{
  pl.m  = m;
  pl.lo = static_cast<int>(int64_t{m} * pl.rank / pl.world);
  pl.hi = static_cast<int>(int64_t{m} * (pl.rank + 1) / pl.world);
  pl.mw = pl.hi - pl.lo;
  pl.q1 = pl.shard ? 0 : pl.lo;
  pl.m1 = pl.shard ? m : pl.mw;
}

/// The batch in the plan's own buffers as one graph.
void capture_batch(index_impl const& ix, plan& pl, cudaStream_t s)
{
  // one eager run first (module loading), then the capture (search.cu:754-786); with several processes
  // the NCCL exchanges between the kernels are captured too (every process replays its graph in the
  // same order, as it would launch the calls)
  run_batch(ix, pl, own_io(pl), s, nullptr);
  OCTEX_CUDA_TRY(cudaStreamSynchronize(s));
  check_tc(pl);
  if (pl.graph != nullptr) {
    cudaGraphExecDestroy(pl.graph);
    pl.graph = nullptr;
  }
  // a large batch of one process in two halves, side by side in the graph (see run_in_place): 10 000 queries of a
  // million rows 850 us one after the other, 810 so
  struct side {
    cudaStream_t s = nullptr;
    ~side()
    {
      if (s != nullptr) cudaStreamDestroy(s);
    }
  } other;
  if (ix.world == 1 && pl.m >= pl.halves_from && !pl.dbg.stats && !pl.dbg.taps)
    OCTEX_CUDA_TRY(cudaStreamCreateWithFlags(&other.s, cudaStreamNonBlocking));
  cudaGraph_t graph = nullptr;
  OCTEX_CUDA_TRY(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
  try {
    if (other.s == nullptr) {
      run_batch(ix, pl, own_io(pl), s, nullptr);
    } else {
      const row_range halves[2] = {{0, (pl.m + 1) / 2}, {(pl.m + 1) / 2, pl.m / 2}};
      OCTEX_CUDA_TRY(cudaEventRecord(pl.join_ev, s));
      OCTEX_CUDA_TRY(cudaStreamWaitEvent(other.s, pl.join_ev, 0));
      run_batch(ix, pl, own_io(pl), s, nullptr, &halves[0]);
      run_batch(ix, pl, own_io(pl), other.s, nullptr, &halves[1]);
      OCTEX_CUDA_TRY(cudaEventRecord(pl.join_ev, other.s));
      OCTEX_CUDA_TRY(cudaStreamWaitEvent(s, pl.join_ev, 0));
    }
  } catch (...) {
    cudaStreamEndCapture(s, &graph);
    if (graph != nullptr) cudaGraphDestroy(graph);
    throw;
  }
  OCTEX_CUDA_TRY(cudaStreamEndCapture(s, &graph));
  const cudaError_t made = cudaGraphInstantiate(&pl.graph, graph, 0);
  cudaGraphDestroy(graph);
  OCTEX_CUDA_TRY(made);
  pl.graph_m = pl.m;
}

auto profile_batch(resources const& res, search_params const& sp, index const& idx, int64_t nq,
                   int64_t k) -> std::vector<float>
{
  auto& ix = idx.impl();
  OCTEX_EXPECTS(nq >= 1 && nq <= std::max(sp.batch, 1),
                "octex: a profiled batch is one batch of queries already on the GPU");
  (void)res;
  auto pl = get_plan(ix, sp, static_cast<int>(nq), static_cast<int>(k));
  std::lock_guard<std::mutex> lock(pl->mu);
  int cur = 0;
  OCTEX_CUDA_TRY(cudaGetDevice(&cur));
  OCTEX_CUDA_TRY(cudaSetDevice(ix.part.device));
  std::vector<cudaEvent_t> marks;
  std::vector<float> ms;
  try {
    set_rows(*pl, static_cast<int>(nq));
    follow_last_batch(*pl, ix.part.stream);
    run_batch(ix, *pl, own_io(*pl), ix.part.stream, &marks);
    OCTEX_CUDA_TRY(cudaStreamSynchronize(ix.part.stream));
    for (size_t i = 1; i < marks.size(); i++) {
      float t = 0.f;
      OCTEX_CUDA_TRY(cudaEventElapsedTime(&t, marks[i - 1], marks[i]));
      ms.push_back(t);
    }
  } catch (...) {
    for (auto e : marks)
      cudaEventDestroy(e);
    cudaSetDevice(cur);
    throw;
  }
  for (auto e : marks)
    cudaEventDestroy(e);
  OCTEX_CUDA_TRY(cudaSetDevice(cur));
  return ms;
}

/// A plan for batches of up to m queries (of exactly m, when several processes share the index).
auto make_plan(index_impl& ix, search_params const& sp, int m, int k, debug_options dbg)
  -> std::shared_ptr<plan>
{
  auto plp  = std::make_shared<plan>();
  plan& pl  = *plp;
  auto& p   = ix.part;
  pl.sp     = sp;
  pl.dbg    = dbg;
  pl.cap    = m;
  pl.k      = k;
  pl.KO     = std::max(sp.starts, k);
  pl.lr     = std::min(sp.read, ix.list_len);
  pl.R1     = sp.rerank;
  pl.R2     = sp.wave_rerank;
  pl.FR     = std::min(sp.final_rerank, pl.KO);
  pl.device = p.device;
  const int D  = static_cast<int>(ix.dim);
  const int sw = ix.sketch_width;
  const int S  = sp.starts;
  const int L  = static_cast<int>(ix.spacings.size());
  // search.cu:637-655
  OCTEX_EXPECTS(sp.read >= 1 && sp.starts >= 1 && sp.waves >= 0,
                "octex: read, starts >= 1 and waves >= 0");
  OCTEX_EXPECTS(sp.waves == 0 || ix.table_len > 0, "octex: waves need the neighbor table");
  OCTEX_EXPECTS(pl.KO <= (sp.sketch_rank ? kernels::kMaxSketchKO : kernels::kMaxRerank),
                "octex: max(starts, k) must be <= 512 (1024 with sketch_rank)");
  OCTEX_EXPECTS(sp.sketch_rank || (sp.rerank >= 1 && sp.rerank <= kernels::kMaxRerank &&
                                   pl.KO + sp.rerank <= kernels::kMaxKeepSort),
                "octex: rerank in [1, 512] and max(starts, k) + rerank <= 1024");
  OCTEX_EXPECTS(sp.sketch_rank || sp.waves == 0 ||
                  (sp.wave_rerank >= 1 && sp.wave_rerank <= kernels::kMaxRerank &&
                   pl.KO + sp.wave_rerank <= kernels::kMaxKeepSort),
                "octex: wave_rerank in [1, 512] and max(starts, k) + wave_rerank <= 1024");
  OCTEX_EXPECTS(!sp.sketch_rank || pl.FR == 0 || (k <= pl.FR && pl.FR <= kernels::kMaxRerank),
                "octex: final_rerank 0 (sketch order) or k <= final_rerank <= 512");
  OCTEX_EXPECTS(sp.waves <= 1 || S * (sp.waves - 1) <= kernels::kMaxExpanded,
                "octex: starts * (waves - 1) <= 6144");
  OCTEX_EXPECTS(int64_t{p.copies} * pl.lr <= kernels::kMaxHash,
                "octex: copies x read too large for the shared-memory hash set");
  OCTEX_EXPECTS(sp.waves == 0 || int64_t{S} * ix.table_len <= kernels::kMaxHash,
                "octex: starts x table_len too large for the shared-memory hash set");
  // slices (search.cu:666-676 of the reference)
  pl.rank  = ix.rank;
  pl.world = ix.world;
  pl.shard = ix.params.mode == placement::shard && ix.world > 1;
  OCTEX_EXPECTS(ix.world == 1 || ix.comm != nullptr,
                "octex: an index shared by several processes needs its communicator first "
                "(octexB200CommInit)");
  OCTEX_EXPECTS(!pl.shard || ix.world * pl.KO <= 4096, "octex: devices * max(starts, k) <= 4096");
  pl.mwmax = (m + ix.world - 1) / ix.world;
  set_rows(pl, m);

  OCTEX_CUDA_TRY(cudaSetDevice(p.device));
  const int m1  = std::max(pl.m1, 1);
  const int wdt = 8 * ix.blocks * p.copies;
  const auto mb = static_cast<size_t>(std::max(pl.mwmax, 1));
  // (the arrays of several processes and of an observed search, and candidates in global memory, come in blocks of their own)
  reserve(pl, p.device,
          {sizeof(float) * m1 * D, sizeof(float) * m1 * sw, sizeof(int2) * m1 * p.copies, sizeof(long long) * m1 * pl.KO,
           sizeof(float) * m1 * pl.KO, (sizeof(long long) + sizeof(float)) * mb * k, sizeof(int) * m1 * S * sp.waves});
  pl.qbuf  = alloc<float>(pl, p.device, int64_t{m1} * D, 0);
  pl.qs    = alloc<float>(pl, p.device, int64_t{m1} * sw);
  pl.use_tc = !dbg.ordered_projection && kernels::project_tc_supported(ix.blocks, p.ldu);
  if (dbg.taps) {
    pl.qh    = alloc<__half>(pl, p.device, int64_t{m1} * p.ldu);
    pl.Y     = alloc<__half>(pl, p.device, int64_t{m1} * wdt);
    pl.codes = alloc<long long>(pl, p.device, int64_t{m1} * p.copies * L);
  }
  // the word a kernel sets when one of its bounded waits (on an mbarrier) ran out
  if (ix.words != nullptr) pl.word = ix.words->take();
  if (pl.word < 0) {
    ix.words = std::make_shared<pinned_words>(p.device);
    pl.word  = ix.words->take();
  }
  pl.words         = ix.words;
  pl.tc_error_host = pl.words->host(pl.word);
  pl.tc_error_dev  = pl.words->device(pl.word);
  if (pl.use_tc) {
    int sms = 0;
    OCTEX_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, p.device));
    kernels::project_tc_setup(pl.tc, p.ut.as<__half>(), p.copies, p.ldu, sms);
  }
  pl.seg   = alloc<int2>(pl, p.device, int64_t{m1} * p.copies);
  pl.si    = alloc<long long>(pl, p.device, int64_t{m1} * pl.KO, 0xff);
  pl.sd    = alloc<float>(pl, p.device, int64_t{m1} * pl.KO);
  const int mwmax = std::max(pl.mwmax, 1);
  // the results of this process's slice: ids [mwmax, k], then distances [mwmax, k], in one block so
  // that one collective moves both
  pl.out_ids = sizeof(long long) * static_cast<size_t>(mwmax) * k;
  pl.out_block = pl.out_ids + sizeof(float) * static_cast<size_t>(mwmax) * k;
  pl.out   = alloc<char>(pl, p.device, static_cast<int64_t>(pl.out_block), 0xff);
  pl.bi    = pl.out.as<long long>();
  pl.bd    = reinterpret_cast<float*>(pl.out.as<char>() + pl.out_ids);
  pl.wsi   = pl.si.as<long long>();
  pl.wsd   = pl.sd.as<float>();
  if (pl.shard) {
    pl.si2    = alloc<long long>(pl, p.device, int64_t{mwmax} * pl.KO, 0xff);
    pl.sd2    = alloc<float>(pl, p.device, int64_t{mwmax} * pl.KO);
    pl.recv_i = alloc<long long>(pl, p.device, int64_t{ix.world} * mwmax * pl.KO, 0xff);
    pl.recv_d = alloc<float>(pl, p.device, int64_t{ix.world} * mwmax * pl.KO, 0);
    pl.wsi    = pl.si2.as<long long>();
    pl.wsd    = pl.sd2.as<float>();
    pl.P_merge = 2;
    while (pl.P_merge < ix.world * pl.KO)
      pl.P_merge <<= 1;
  }
  if (ix.world > 1) {
    pl.gathered = alloc<char>(pl, p.device, static_cast<int64_t>(pl.out_block) * ix.world, 0xff);
  }
  if (sp.waves > 0) pl.done = alloc<int>(pl, p.device, int64_t{m1} * S * sp.waves, 0xff);
  if (dbg.stats) {
    pl.stats  = alloc<long long>(pl, p.device, int64_t{m1} * 8, 0);
    pl.phase1 = alloc<long long>(pl, p.device, int64_t{m1} * 8, 0);
    pl.phase2 = alloc<long long>(pl, p.device, int64_t{m1} * 8, 0);
  }
  if (dbg.taps) {
    pl.tap_cap  = p.copies * pl.lr;
    pl.tap_cand = alloc<int>(pl, p.device, int64_t{m1} * pl.tap_cap, 0xff);
    pl.tap_dist = alloc<float>(pl, p.device, int64_t{m1} * pl.tap_cap, 0);
    pl.tap_n    = alloc<int>(pl, p.device, m1, 0);
    pl.kept1_i  = alloc<long long>(pl, p.device, int64_t{m1} * pl.KO, 0xff);
    pl.kept1_d  = alloc<float>(pl, p.device, int64_t{m1} * pl.KO, 0);
  }

  // first round: lists of this process's copies
  auto& r1       = pl.r1;
  r1.m           = pl.m1;
  r1.nseg        = p.copies;
  r1.seg         = pl.seg.as<int2>();
  r1.lists       = p.lists.as<int>();
  r1.stride      = p.stride;
  r1.lr          = pl.lr;
  r1.sketch      = p.sketch.as<signed char>();
  r1.sketch_norm = p.sketch_norm.as<float>();
  r1.scale       = p.scale.as<float>();
  r1.qs          = pl.qs.as<float>();
  r1.sw          = sw;
  r1.vectors     = p.vectors.as<__half>();
  r1.D           = D;
  r1.Q           = pl.qbuf.as<float>();
  r1.R           = pl.R1;
  r1.KO          = pl.KO;
  r1.sketch_rank = sp.sketch_rank ? 1 : 0;
  r1.sketch_map  = map_of(ix, p.sketch_rows);
  r1.vector_map  = map_of(ix, p.vector_rows);
  r1.si          = pl.si.as<long long>();
  r1.sd          = pl.sd.as<float>();
  r1.stats       = pl.stats.as<long long>();
  r1.phase       = pl.phase1.as<long long>();
  if (dbg.taps) {
    r1.tap_cand = pl.tap_cand.as<int>();
    r1.tap_dist = pl.tap_dist.as<float>();
    r1.tap_n    = pl.tap_n.as<int>();
    r1.tap_cap  = pl.tap_cap;
  }
  // sketch rows of this GPU's own memory (not the host tier, not dealt over GPUs) plus their constants
  const int64_t sketch_bytes = (p.sketch.host || p.sketch_rows.on) ? 0 : static_cast<int64_t>(p.sketch.size + p.sketch_norm.size);
  size_round(pl, r1, p.copies * pl.lr, false, 0, p.device, sketch_bytes, ix.n, !p.vectors.host);
  // waves: table rows of the start points
  if (sp.waves > 0) {
    auto& r2       = pl.r2;
    r2             = kernels::round_args{};
    r2.m           = pl.mw;
    r2.nseg        = S;
    r2.table       = p.table.as<int>();
    r2.table_len   = ix.table_len;
    r2.table_map   = map_of(ix, p.table_rows);
    r2.sketch_map  = r1.sketch_map;
    r2.vector_map  = r1.vector_map;
    r2.done        = pl.done.as<int>();
    r2.done_stride = S * sp.waves;
    r2.sketch      = r1.sketch;
    r2.sketch_norm = r1.sketch_norm;
    r2.scale       = r1.scale;
    r2.qs          = r1.qs + static_cast<size_t>(pl.lo - pl.q1) * sw;
    r2.sw          = sw;
    r2.vectors     = r1.vectors;
    r2.D           = D;
    r2.Q           = r1.Q + static_cast<size_t>(pl.lo - pl.q1) * D;
    r2.R           = pl.R2;
    r2.KO          = pl.KO;
    r2.sketch_rank = r1.sketch_rank;
    r2.si          = pl.wsi;
    r2.sd          = pl.wsd;
    r2.stats       = r1.stats;
    r2.phase       = pl.phase2.as<long long>();
    size_round(pl, r2, S * ix.table_len, true, S * std::max(sp.waves - 1, 0), p.device, sketch_bytes, ix.n, !p.vectors.host);
  }
  kernels::round_allow_smem();
  {
    // Kernels of the two halves of a batch run side by side, one's under the end of the other's, where there are
    // more query blocks than the multiprocessors hold of its heaviest round (twice as many where they hold one
    // each) and a million entries to gather. us a search, whole and in halves: a million rows, eight blocks each, 1 000
    // queries 161 and 176, 1 200 216 and 208, 2 500 307 and 277, 10 000 861 and 831; four blocks each, 500 195 and
    // 194, 700 264 and 232, 4 000 982 and 930; two, 300 473 and 448, 1 200 1 212 and 1 094, 10 000 8 143 and 8 021; one,
    // 200 527 and 587, 400 747 and 681, 2 500 3 556 and 3 432. A small index with 32 entries a query, 1 200 55 and
    // 58, 3 000 65 and 66; 256 entries, 1 300 110 and 109; 1 088, 1 200 117 and 116, 1 500 124 and 116.
    int64_t held = 0, entries = 0;
    for (auto const* r : {&r1, &pl.r2}) {
      if (r == &pl.r2 && sp.waves == 0) continue;
      const auto per_sm = std::min<int64_t>(static_cast<int64_t>(blocks_of(*r)), 1024 / r->threads);
      held              = held == 0 ? per_sm : std::min(held, per_sm);
      entries += int64_t{r->nmax} * (r == &r1 ? 1 : sp.waves);
    }
    pl.entries     = entries;
    pl.halves_from = std::max(held >= 2 ? held * r1.sms + 1 : int64_t{2} * r1.sms, (1 << 20) / entries);
  }

  OCTEX_CUDA_TRY(cudaEventCreateWithFlags(&pl.done_ev, cudaEventDisableTiming));
  OCTEX_CUDA_TRY(cudaEventCreateWithFlags(&pl.join_ev, cudaEventDisableTiming));
  OCTEX_CUDA_TRY(cudaDeviceSynchronize());  // the buffers are filled on the default stream
  if (ix.world > 1) capture_batch(ix, pl, p.stream);
  return plp;
}

namespace {

/// The name of a configuration. One process: a plan serves every batch it has room for. Several: their
/// slices and exchanges depend on the number of queries.
auto plan_key(index_impl const& ix, search_params const& sp, int m, int k, debug_options dbg) -> std::string
{
  return std::to_string(ix.world > 1 ? m : 0) + "/" + std::to_string(k) + "/" + std::to_string(sp.read) + "/" +
         std::to_string(sp.starts) + "/" + std::to_string(sp.waves) + "/" + std::to_string(sp.rerank) + "/" +
         std::to_string(sp.wave_rerank) + "/" + std::to_string(sp.sketch_rank) + "/" +
         std::to_string(sp.final_rerank) + "/" + std::to_string(dbg.stats) + std::to_string(dbg.taps) +
         std::to_string(dbg.ordered_projection);
}
auto lane_name(std::string const& key, int lane) -> std::string { return lane == 0 ? key : key + "#" + std::to_string(lane); }

}  // namespace

auto get_plan(index_impl& ix, search_params const& sp, int m, int k, int lane) -> std::shared_ptr<plan>
{
  const debug_options dbg = ix_debug(ix);
  const std::string key   = plan_key(ix, sp, m, k, dbg);
  std::lock_guard<std::mutex> lock(ix.mu);
  // one cached configuration: the previous buffers and graphs go before the new ones come
  // (search.cu:807-812); a configuration has one plan per lane (see search_impl)
  if (ix.plans.find(key) == ix.plans.end()) ix.plans.clear();
  const std::string name = lane_name(key, lane);
  auto& pl               = ix.plans[name];
  if (pl == nullptr || pl->cap < m) {
    pl.reset();
    try {
      pl = make_plan(ix, sp, m, k, dbg);
    } catch (...) {
      ix.plans.erase(name);
      throw;
    }
  }
  return pl;
}

namespace {

/// True when a kernel of this GPU and the copy engines reach p directly (page-locked or device memory).
auto device_reaches(const void* p) -> bool
{
  cudaPointerAttributes at{};
  if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return at.type != cudaMemoryTypeUnregistered;
}

/// True when p is memory of this GPU itself and on a boundary of `align` bytes: what the kernels of a
/// search may load and store themselves. Another GPU's memory is not mapped here, managed and
/// page-locked memory is better copied once than read over the bus by every block.
auto own_memory(const void* p, int device, size_t align) -> bool
{
  cudaPointerAttributes at{};
  if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return at.type == cudaMemoryTypeDevice && at.device == device && reinterpret_cast<uintptr_t>(p) % align == 0;
}

/// Page-locked staging of at least `bytes`, kept with the plan.
void* staging(dbuf& b, int device, size_t bytes)
{
  if (b.size < bytes) b = dbuf::pinned(device, bytes);
  return b.ptr;
}

/// The event of the index for streams of device `dev`, the current one; ix.start_mu guards it.
auto start_event(index_impl& ix, int dev) -> cudaEvent_t
{
  if (ix.start_ev == nullptr || ix.start_dev != dev) {
    if (ix.start_ev != nullptr) cudaEventDestroy(ix.start_ev);
    ix.start_ev = nullptr;
    OCTEX_CUDA_TRY(cudaEventCreateWithFlags(&ix.start_ev, cudaEventDisableTiming));
    ix.start_dev = dev;
  }
  return ix.start_ev;
}

/// The stream of the second lane, made when first needed (its device is current; ix.start_mu guards it).
auto second_stream(index_impl& ix) -> cudaStream_t
{
  auto& p = ix.part;
  if (p.second == nullptr) OCTEX_CUDA_TRY(cudaStreamCreateWithFlags(&p.second, cudaStreamNonBlocking));
  return p.second;
}

/// Queries of the batches a call is cut into. Two are halves, since nothing is left to run under the end
/// of the second: 10 100 queries, batch 10 000, 600 us against 650 as 10 000 and 100, and 12 345 from host
/// memory 1 097 against 1 213. Three and more are whole batches and a rest (1 067 queries, batch 400, 256
/// start points and three waves: 646 us against 706 in thirds).
auto batch_rows(int64_t nq, int batch) -> int
{
  const int64_t most = std::max(batch, 1);
  return static_cast<int>(nq <= most ? nq : nq <= 2 * most ? (nq + 1) / 2 : most);
}

/// The plans of a call: one, or one per lane.
using lane_plans = std::array<std::shared_ptr<plan>, 2>;

/// The plans of a call by one process. The first has room for a whole batch, also when the call is cut
/// into halves: a resident search takes the whole batch from it (gather_resident).
auto plans_of(index_impl& ix, search_params const& sp, int lanes, int64_t nq, int64_t k) -> lane_plans
{
  lane_plans lane;
  for (int l = 0; l < lanes; l++)
    lane[l] = get_plan(ix, sp, l == 0 ? static_cast<int>(std::min<int64_t>(nq, std::max(sp.batch, 1))) : batch_rows(nq, sp.batch),
                       static_cast<int>(k), l);
  return lane;
}

/// The stream of the second half of a batch of n queries, if it goes in halves: not while s is captured (so this stream
/// never is, whatever other threads capture), nor under observation. Its device is current, ix.start_mu is held.
auto half_stream(index_impl& ix, plan const& pl, int n, cudaStream_t s) -> cudaStream_t
{
  if (n < pl.halves_from || pl.dbg.stats || pl.dbg.taps || capturing(s)) return nullptr;
  auto& p = ix.part;
  if (p.half == nullptr) OCTEX_CUDA_TRY(cudaStreamCreateWithFlags(&p.half, cudaStreamNonBlocking));
  return p.half;
}

/// What s holds from now on comes after the half of a batch queued on `other`. A half is joined as well when the
/// batch could not be queued whole; where not even that can be queued the host waits, so that no call returns with the
/// caller's arrays in use on a stream that the caller does not know.
struct half_join {
  cudaEvent_t ev;
  cudaStream_t s, other;
  bool open = true;
  half_join(plan const& pl, cudaStream_t on, cudaStream_t half) : ev(pl.join_ev), s(on), other(half) {}
  half_join(half_join const&) = delete;
  void close()
  {
    OCTEX_CUDA_TRY(cudaEventRecord(ev, other));
    OCTEX_CUDA_TRY(cudaStreamWaitEvent(s, ev, 0));
    open = false;
  }
  ~half_join()
  {
    if (!open || (cudaEventRecord(ev, other) == cudaSuccess && cudaStreamWaitEvent(s, ev, 0) == cudaSuccess)) return;
    cudaStreamSynchronize(other);
    cudaGetLastError();  // the error to report is on its way
  }
};

/// A batch of n queries in device memory on s; in two halves where that pays: the second runs on the other stream,
/// from where s is now, and s goes on when it is done.
void run_in_place(index_impl& ix, plan& pl, batch_io const& io, int n, cudaStream_t s)
{
  std::unique_lock<std::mutex> one_start(ix.start_mu);
  cudaStream_t other = half_stream(ix, pl, n, s);
  if (other == nullptr) {
    one_start.unlock();
    run_batch(ix, pl, io, s, nullptr);
    return;
  }
  OCTEX_CUDA_TRY(cudaEventRecord(start_event(ix, ix.part.device), s));
  OCTEX_CUDA_TRY(cudaStreamWaitEvent(other, ix.start_ev, 0));
  one_start.unlock();
  half_join join(pl, s, other);
  const row_range halves[2] = {{0, (n + 1) / 2}, {(n + 1) / 2, n / 2}};
  run_batch(ix, pl, io, s, nullptr, &halves[0]);
  run_batch(ix, pl, io, other, nullptr, &halves[1]);
  join.close();
}

/// The next batch of a call on a plan: n queries from row b0 of it on.
void set_batch(plan& pl, unsigned long long call, int64_t b0, int n)
{
  set_rows(pl, n);
  pl.call  = call;
  pl.first = b0;
  pl.held  = n;
}

/// The m queries a resident search of the plan repeats, of which it may hold fewer: what the other lane
/// of the same call holds behind them comes over, the rest is filled with copies of the first query
/// (search.cu:870-883 of the reference). Queued on s; the plan's lock is held.
void gather_resident(index_impl& ix, search_params const& sp, plan& pl, int m, int k, cudaStream_t s)
{
  if (pl.held >= m || pl.held == 0) return;
  std::shared_ptr<plan> other;
  {
    std::lock_guard<std::mutex> lock(ix.mu);
    const auto at = ix.plans.find(lane_name(plan_key(ix, sp, m, k, pl.dbg), 1));
    if (at != ix.plans.end()) other = at->second;
  }
  const auto D = static_cast<size_t>(ix.dim);
  if (other != nullptr) {
    std::lock_guard<std::mutex> lock(other->mu);
    if (other->call == pl.call && other->first == pl.first + pl.held) {
      const int n = std::min(other->held, m - pl.held);
      follow_last_batch(*other, s);
      OCTEX_CUDA_TRY(cudaMemcpyAsync(pl.qbuf.as<float>() + pl.held * D, other->qbuf.ptr, sizeof(float) * n * D,
                                     cudaMemcpyDeviceToDevice, s));
      mark_last_batch(*other, s);  // its next batch comes after the copy
      pl.held += n;
    }
  }
  kernels::pad_rows(pl.qbuf.as<float>(), pl.held, m, static_cast<int>(D), s);
}

/// A search by one process with queries and results in the memory of its GPU: the batches run from the
/// caller's arrays and into them. One batch stays on the caller's stream; several alternate between it
/// and a second one, each with a plan of its own: the rounds of a batch end in blocks that leave
/// multiprocessors idle, whatever its size. 200 000 rows x 128, one stream and two: 3 x 300 queries with
/// 256 start points and three waves 830 and 636 us, 10 x 1 000 queries 1 016 and 727, 3 x 10 000
/// 1 787 and 1 700.
auto search_device(index_impl& ix, search_params const& sp, int lanes, cudaStream_t caller, const float* queries,
                   int64_t nq, int64_t* neighbors, float* distances, int64_t k) -> lane_plans
{
  const int m                   = batch_rows(nq, sp.batch);
  const unsigned long long call = ++ix.calls;
  const lane_plans lane         = plans_of(ix, sp, lanes, nq, k);
  std::unique_lock<std::mutex> lock0(lane[0]->mu), lock1;
  if (lanes > 1) lock1 = std::unique_lock<std::mutex>(lane[1]->mu);
  cudaStream_t stream[2] = {caller, caller};
  if (lanes > 1) {
    std::lock_guard<std::mutex> one_start(ix.start_mu);
    stream[1] = second_stream(ix);
    OCTEX_CUDA_TRY(cudaEventRecord(start_event(ix, ix.part.device), caller));
    OCTEX_CUDA_TRY(cudaStreamWaitEvent(stream[1], ix.start_ev, 0));
  }
  for (int l = 0; l < lanes; l++) {
    // a search with device outputs returns before its kernels ran; had one of them given up, the
    // word is still set and this is the first host code to see it
    check_tc(*lane[l]);
    follow_last_batch(*lane[l], stream[l]);
  }
  auto run = [&](int l, int64_t b0, int n) {
    set_batch(*lane[l], call, b0, n);
    const batch_io io{queries + b0 * ix.dim, reinterpret_cast<long long*>(neighbors + b0 * k), distances + b0 * k};
    if (lanes == 1)
      run_in_place(ix, *lane[l], io, n, stream[l]);
    else
      run_batch(ix, *lane[l], io, stream[l], nullptr);
  };
  auto close = [&](int l, bool) {
    mark_last_batch(*lane[l], stream[l]);
    if (l == 0) return;
    OCTEX_CUDA_TRY(cudaEventRecord(lane[l]->join_ev, stream[l]));
    OCTEX_CUDA_TRY(cudaStreamWaitEvent(caller, lane[l]->join_ev, 0));
  };
  each_batch(nq, m, lanes, run, close);
  return lane;
}

/// Queries of a batch in ordinary host memory go through staging of the plan below this many bytes: a
/// memcpy and a copy that need not be waited for. Above it the driver's copy from ordinary memory, which
/// stages piece by piece while the pieces before cross the bus, is the faster one, although the call
/// waits in it. us a call, staged and not: 100 queries x 128 (51 KB) 86 and 87, three batches of them 174
/// and 212, 500 x 128 (256 KB) 122 and 125, 3 x 800 (410 KB) 354 and 341, 1 000 x 128 (512 KB) 173 and 170,
/// 200 x 960 (768 KB) 239 and 229, 2 000 x 960 1 268 and 1 101, 10 000 x 128 1 090 and 987.
constexpr size_t kStagedQueries = size_t{384} << 10;

/// Results in ordinary host memory: true when they are made on the GPU and copied by the driver, false when
/// the last kernel stores them through to staging. The stores cross the bus under the kernel's other
/// work where it has enough of it; a round that gathers few entries per result ends waiting for them.
/// 10 000 queries x 100 results (12 MB), stored and copied: 2 048 entries a query 1 721 and 1 797 us, 256
/// entries a query 1 286 and 1 168; with 5 000 queries 690 and 659, 3 000 (3.6 MB) 440 and 437, 2 000 317 and 321.
auto copies_results(plan const& pl, int m) -> bool
{
  constexpr size_t kLarge = size_t{4} << 20;
  const size_t bytes      = (sizeof(int64_t) + sizeof(float)) * static_cast<size_t>(m) * pl.k;
  const int entries       = pl.sp.waves > 0 ? pl.r2.nmax : pl.r1.nmax;
  return bytes >= kLarge && entries < 8 * pl.k;
}

/// Entries a batch in ordinary host memory gathers from which on it goes in two halves: the call waits twice in the
/// copies of its queries then, under kernels that have to be long enough. us a call, whole and in halves: 3.3
/// million (3 000 queries of a small index) 269 and 297, 3.7 (1 200 x 128) 292 and 293, 6.1 375 and 365, 6.5 482 and
/// 451, 7.7 457 and 406, 15 743 and 745, 18 859 and 824, 31 1 414 and 1 295.
constexpr int64_t kCopiedEntries = int64_t{1} << 22;

/// A search by one process with queries and results that are not all memory of its GPU (host memory,
/// another GPU's): the copies are queued around the kernels. Several batches alternate between two
/// lanes, each a plan on a stream of its own: the copies of one batch run under the kernels of the
/// other. So do the halves of a batch that goes in two, on two streams with one plan. Page-locked arrays
/// are copied from and to directly; ordinary ones pass through page-locked staging of the plan where that
/// is faster (kStagedQueries, copies_results).
void search_copied(index_impl& ix, search_params const& sp, int lanes, cudaStream_t caller, int cur, const float* queries,
                   int64_t nq, int64_t* neighbors, float* distances, int64_t k, bool host_out)
{
  auto& p                       = ix.part;
  const int D                   = static_cast<int>(ix.dim);
  int m                         = batch_rows(nq, sp.batch);
  const unsigned long long call = ++ix.calls;
  lane_plans lane               = plans_of(ix, sp, lanes, nq, k);
  std::unique_lock<std::mutex> lock0(lane[0]->mu), lock1;
  if (lanes > 1) lock1 = std::unique_lock<std::mutex>(lane[1]->mu);
  cudaStream_t stream[2] = {p.stream, p.second};
  for (int l = 0; l < lanes; l++) {
    check_tc(*lane[l]);
    follow_last_batch(*lane[l], stream[l]);
  }
  bool halves = false;  // of the one batch there is, lane l's from row l * m of the plan's arrays on
  if (lanes == 1 && nq == m) {
    stream[1] = nullptr;
    std::lock_guard<std::mutex> one_start(ix.start_mu);
    // (a copy of results to ordinary memory would hold up the second half)
    if (!(host_out && (copies_results(*lane[0], m) || m * lane[0]->entries < kCopiedEntries)))
      stream[1] = half_stream(ix, *lane[0], m, stream[0]);
    halves = stream[1] != nullptr;
  }
  if (halves) {
    lanes     = 2;
    m         = (m + 1) / 2;
    lane[1]   = lane[0];
    set_batch(*lane[0], call, 0, static_cast<int>(nq));
    OCTEX_CUDA_TRY(cudaEventRecord(lane[0]->join_ev, stream[0]));
    OCTEX_CUDA_TRY(cudaStreamWaitEvent(stream[1], lane[0]->join_ev, 0));
  }
  const bool stage_in  = host_out && sizeof(float) * static_cast<size_t>(m) * D < kStagedQueries && !device_reaches(queries);
  const bool stage_out = host_out && !(lanes == 1 && copies_results(*lane[0], m)) &&
                         !(device_reaches(neighbors) && device_reaches(distances));
  struct pending {
    int64_t b0 = 0;
    int n      = 0;
  } out[2];
  // results of the last batch of a lane from its staging to the caller's arrays
  auto deliver = [&](int l) {
    if (out[l].n == 0) return;
    OCTEX_CUDA_TRY(cudaStreamSynchronize(stream[l]));
    plan& w            = *lane[l];
    const size_t cnt   = static_cast<size_t>(out[l].n) * k;
    const size_t from  = halves ? static_cast<size_t>(l) * m * k : 0;
    const auto* dist   = reinterpret_cast<const float*>(w.stage_out.as<int64_t>() + static_cast<size_t>(w.cap) * k);
    std::memcpy(neighbors + out[l].b0 * k, w.stage_out.as<int64_t>() + from, cnt * sizeof(int64_t));
    std::memcpy(distances + out[l].b0 * k, dist + from, cnt * sizeof(float));
    out[l].n = 0;
  };
  int64_t batch = 0;
  auto run      = [&](int l, int64_t b0, int n) {
    plan& w            = *lane[l];
    cudaStream_t s     = stream[l];
    const size_t bytes = sizeof(float) * static_cast<size_t>(n) * D;
    const row_range part{halves ? l * m : 0, n};
    float* own_q = w.qbuf.as<float>() + static_cast<size_t>(part.first) * D;
    if (stage_out) deliver(l);  // the lane's staging is free again, its queries too
    const void* src = queries + b0 * D;
    if (stage_in) {
      if (!stage_out && batch >= lanes) OCTEX_CUDA_TRY(cudaStreamSynchronize(s));
      float* pin = static_cast<float*>(staging(w.stage_q, p.device, sizeof(float) * static_cast<size_t>(w.cap) * D)) +
                   static_cast<size_t>(part.first) * D;
      std::memcpy(pin, src, bytes);
      src = pin;
    }
    OCTEX_CUDA_TRY(cudaMemcpyAsync(own_q, src, bytes, cudaMemcpyDefault, s));
    if (!halves) set_batch(w, call, b0, n);
    batch_io io = own_io(w);
    if (stage_out) {
      // the last kernel writes through to host memory
      auto* pin = static_cast<char*>(staging(w.stage_out, p.device, (sizeof(int64_t) + sizeof(float)) * static_cast<size_t>(w.cap) * k));
      io.ids    = reinterpret_cast<long long*>(pin);
      io.dist   = reinterpret_cast<float*>(pin + sizeof(int64_t) * static_cast<size_t>(w.cap) * k);
    }
    run_batch(ix, w, io, s, nullptr, halves ? &part : nullptr);
    if (stage_out) {
      out[l].b0 = b0;
      out[l].n  = n;
    } else {
      const int64_t from = int64_t{part.first} * k;
      OCTEX_CUDA_TRY(cudaMemcpyAsync(neighbors + b0 * k, w.bi + from, sizeof(int64_t) * n * k, cudaMemcpyDefault, s));
      OCTEX_CUDA_TRY(cudaMemcpyAsync(distances + b0 * k, w.bd + from, sizeof(float) * n * k, cudaMemcpyDefault, s));
    }
    batch++;
  };
  auto close = [&](int l, bool failed) {
    if (halves && l == 0) return;
    if (halves) {  // what the plan's last batch is ends on the first stream
      half_join(*lane[0], stream[0], stream[1]).close();
      l = 0;
    }
    mark_last_batch(*lane[l], stream[l]);
    if (host_out) {
      // nothing may still be on its way from or to the caller's arrays or the staging
      if (failed) OCTEX_CUDA_TRY(cudaStreamSynchronize(stream[l]));
      return;
    }
    OCTEX_CUDA_TRY(cudaEventRecord(lane[l]->join_ev, stream[l]));
    OCTEX_CUDA_TRY(cudaSetDevice(cur));
    OCTEX_CUDA_TRY(cudaStreamWaitEvent(caller, lane[l]->join_ev, 0));
    OCTEX_CUDA_TRY(cudaSetDevice(p.device));
  };
  each_batch(nq, m, lanes, run, close);
  if (!host_out) return;
  if (stage_out && lanes > 1) deliver(static_cast<int>(batch % lanes));  // the older of the two first
  for (int l = 0; l < lanes; l++) {
    if (stage_out) deliver(l);
    OCTEX_CUDA_TRY(cudaStreamSynchronize(stream[l]));
    check_tc(*lane[l]);
  }
}

}  // namespace

auto search_in_place(index_impl const& ix, const float* queries, const int64_t* neighbors, const float* distances) -> bool
{
  int cur = 0;
  OCTEX_CUDA_TRY(cudaGetDevice(&cur));
  const int device = ix.part.device;
  return ix.world == 1 && cur == device && own_memory(queries, device, alignof(float)) &&
         own_memory(neighbors, device, alignof(int64_t)) && own_memory(distances, device, alignof(float));
}

void search_impl(resources const& res,
                 search_params const& sp,
                 index const& idx,
                 const float* queries,
                 int64_t nq,
                 int64_t qdim,
                 int64_t* neighbors,
                 float* distances,
                 int64_t k,
                 bool host_out,
                 bool resident,
                 bool wait,
                 int max_lanes)
{
  auto& ix = idx.impl();
  OCTEX_EXPECTS(qdim == ix.dim, "octex: query dimension differs from the index");
  OCTEX_EXPECTS(k >= 1, "octex: k >= 1");
  if (nq == 0) return;
  int cur = 0;
  OCTEX_CUDA_TRY(cudaGetDevice(&cur));
  cudaStream_t caller = res.stream;
  auto& p             = ix.part;
  // streams: a second one for the batches of one process, unless the plan keeps observations
  const debug_options dbg = ix_debug(ix);
  const int lanes = ix.world == 1 && !resident && nq > std::max(sp.batch, 1) && !dbg.stats && !dbg.taps ? max_lanes : 1;
  if (!resident && !host_out && search_in_place(ix, queries, neighbors, distances)) {
    const lane_plans used = search_device(ix, sp, lanes, caller, queries, nq, neighbors, distances, k);
    if (wait) {
      OCTEX_CUDA_TRY(cudaStreamSynchronize(caller));
      for (auto const& pl : used)
        if (pl != nullptr) check_tc(*pl);
    }
    return;
  }
  // the work of this call starts after what the caller queued on its stream (search.cu:841-848): an
  // event of the index, on the device of the caller's stream, which is the current one
  struct back_to {
    int device;
    ~back_to() { cudaSetDevice(device); }
  } back{cur};
  std::unique_lock<std::mutex> one_start(ix.start_mu);
  const bool busy = capturing(caller) || cudaStreamQuery(caller) != cudaSuccess;
  if (busy) {
    cudaGetLastError();  // "not ready" is no failure
    OCTEX_CUDA_TRY(cudaEventRecord(start_event(ix, cur), caller));
  }
  OCTEX_CUDA_TRY(cudaSetDevice(p.device));
  if (lanes > 1) second_stream(ix);
  if (busy) {
    OCTEX_CUDA_TRY(cudaStreamWaitEvent(p.stream, ix.start_ev, 0));
    if (lanes > 1) OCTEX_CUDA_TRY(cudaStreamWaitEvent(p.second, ix.start_ev, 0));
  }
  one_start.unlock();
  if (ix.world == 1 && !resident) {
    search_copied(ix, sp, lanes, caller, cur, queries, nq, neighbors, distances, k, host_out);
    if (wait && !host_out) OCTEX_CUDA_TRY(cudaStreamSynchronize(caller));
    return;
  }
  // resident queries, or batches in which processes exchange: one lane, one graph per batch
  const int m = static_cast<int>(std::min<int64_t>(std::max(sp.batch, 1), nq));
  auto pl     = get_plan(ix, sp, m, static_cast<int>(k));
  plan& w     = *pl;
  const int D = static_cast<int>(ix.dim);
  std::unique_lock<std::mutex> lock0(w.mu);
  cudaStream_t s = p.stream;
  check_tc(w);
  follow_last_batch(w, s);
  if (ix.world == 1) {
    set_rows(w, m);
    gather_resident(ix, sp, w, m, static_cast<int>(k), s);
    if (sp.use_graph && (w.graph == nullptr || w.graph_m != m)) capture_batch(ix, w, s);
  }
  auto run = [&](int, int64_t b0, int n) {
    if (!resident) {
      // rows [q1, q1 + m1) of the batch, the part beyond its end filled with copies of a row
      // (search.cu:870-883)
      int have = std::clamp(n - w.q1, 0, w.m1);
      if (have > 0) {
        OCTEX_CUDA_TRY(cudaMemcpyAsync(w.qbuf.ptr, queries + (b0 + w.q1) * D, sizeof(float) * have * D,
                                       cudaMemcpyDefault, s));
      } else if (w.m1 > 0) {
        OCTEX_CUDA_TRY(cudaMemcpyAsync(w.qbuf.ptr, queries + b0 * D, sizeof(float) * D, cudaMemcpyDefault, s));
        have = 1;
      }
      if (have < w.m1) kernels::pad_rows(w.qbuf.as<float>(), have, w.m1, D, s);
    }
    if (sp.use_graph && w.graph != nullptr)
      OCTEX_CUDA_TRY(cudaGraphLaunch(w.graph, s));
    else
      run_batch(ix, w, own_io(w), s, nullptr);  // use_graph = false
    if (!resident) {
      // the gathered results: block r holds the rows [lo_r, hi_r) of the batch
      for (int r = 0; r < w.world; r++) {
        const int lo_r = static_cast<int>(int64_t{m} * r / w.world);
        const int hi_r = static_cast<int>(int64_t{m} * (r + 1) / w.world);
        const int rows = std::clamp(n - lo_r, 0, hi_r - lo_r);
        if (rows == 0) continue;
        const char* block = w.gathered.as<char>() + static_cast<size_t>(r) * w.out_block;
        OCTEX_CUDA_TRY(cudaMemcpyAsync(neighbors + (b0 + lo_r) * k, block, sizeof(int64_t) * rows * k,
                                       cudaMemcpyDefault, s));
        OCTEX_CUDA_TRY(cudaMemcpyAsync(distances + (b0 + lo_r) * k, block + w.out_ids, sizeof(float) * rows * k,
                                       cudaMemcpyDefault, s));
      }
    }
  };
  auto close = [&](int, bool) {
    mark_last_batch(w, s);
    OCTEX_CUDA_TRY(cudaEventRecord(w.join_ev, s));
    OCTEX_CUDA_TRY(cudaSetDevice(cur));
    OCTEX_CUDA_TRY(cudaStreamWaitEvent(caller, w.join_ev, 0));
  };
  each_batch(nq, m, 1, run, close);
  if (host_out || wait) {
    OCTEX_CUDA_TRY(cudaStreamSynchronize(caller));
    check_tc(w);
  }
}

}  // namespace detail

void search(resources const& res, search_params const& params, index const& idx,
            host_matrix_view<const float> queries, host_matrix_view<int64_t> neighbors,
            host_matrix_view<float> distances)
{
  OCTEX_EXPECTS(neighbors.rows == queries.rows && distances.rows == queries.rows &&
                  distances.cols == neighbors.cols,
                "octex: output shapes");
  detail::search_impl(res, params, idx, queries.data, queries.rows, queries.cols, neighbors.data,
                      distances.data, neighbors.cols, true, false);
}

void search(resources const& res, search_params const& params, index const& idx,
            device_matrix_view<const float> queries, device_matrix_view<int64_t> neighbors,
            device_matrix_view<float> distances)
{
  OCTEX_EXPECTS(neighbors.rows == queries.rows && distances.rows == queries.rows &&
                  distances.cols == neighbors.cols,
                "octex: output shapes");
  detail::search_impl(res, params, idx, queries.data, queries.rows, queries.cols, neighbors.data,
                      distances.data, neighbors.cols, false, false);
}

}  // namespace octex_b200
