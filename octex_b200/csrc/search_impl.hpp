// Buffers and graph of one batch shape and one set of search parameters (the reference's
// plan / gpu_plan, cpp/src/neighbors/octex/search.cu:35-80 of hpdic/octex, for one GPU).
#pragma once

#include "index_impl.hpp"
#include "kernels.hpp"

#include <mutex>
#include <vector>

namespace octex_b200::detail {

struct plan {
  search_params sp;
  debug_options dbg;
  int device = 0;
  // m: queries of the last batch (with several processes: of every batch); cap: the most a batch may
  // have, what the buffers are sized for
  int m = 0, cap = 0, k = 0, KO = 0, lr = 0, R1 = 0, R2 = 0, FR = 0;
  // Who answers what in a batch of m rows when `world` processes share the index
  // (search.cu:666-676 of the reference, per GPU there, per process here): the first round runs on
  // rows [q1, q1 + m1) — all m rows when the copies are sharded, the own slice otherwise — and the
  // waves on the own slice [lo, hi).
  int rank = 0, world = 1;
  bool shard = false;
  int m1 = 0, q1 = 0, lo = 0, hi = 0, mw = 0, mwmax = 0;
  dbuf si2, sd2;        // shard: kept list of the own slice after the cross-process merge
  dbuf recv_i, recv_d;  // shard: [world, mwmax, KO] first-round kept lists of every process
  dbuf out;             // results of this process's slice: ids [mwmax, k], then distances [mwmax, k]
  dbuf gathered;        // world > 1: the out blocks of every process
  size_t out_block = 0, out_ids = 0;  // bytes of a block and of its ids
  long long* bi = nullptr;            // the two arrays inside out
  float* bd     = nullptr;
  long long* wsi = nullptr;  // kept list the waves work on [mw, KO]
  float* wsd     = nullptr;
  int P_merge    = 0;   // keys sorted by the cross-process merge (power of two >= world * KO)
  dbuf qbuf, qh, qs, Y, codes, seg, si, sd, done, stats, phase1, phase2;
  dbuf tap_cand, tap_dist, tap_n, kept1_i, kept1_d;
  bool use_tc = false;          // tensor-core projection with the decode in its epilogue
  kernels::project_tc_plan tc;  // its tensor maps
  std::shared_ptr<pinned_words> words;  // a word of the index, non-zero when a bounded wait in a kernel ran out
  int word           = -1;
  int* tc_error_host = nullptr;
  int* tc_error_dev  = nullptr;
  int tap_cap = 0;
  std::vector<dbuf> scratch_cand, scratch_dist;
  kernels::round_args r1, r2;
  cudaGraphExec_t graph = nullptr;  // of a batch of graph_m queries in the plan's own buffers
  int graph_m           = 0;
  cudaEvent_t done_ev   = nullptr;  // the end of the plan's last batch
  cudaEvent_t join_ev   = nullptr;  // the same for the caller's stream to wait for, also while it is captured
  // the queries of the last call that qbuf still holds, [first, first + held) of it, and which call that was
  int64_t first              = 0;
  int held                   = 0;
  unsigned long long call    = 0;
  // the stream done_ev was recorded on (cudaStreamGetId): a batch on another one waits for it first
  unsigned long long last_stream = 0;
  bool used                      = false;
  int64_t entries       = 0;  // list and table entries that a query gathers at most
  int64_t halves_from   = 0;  // queries from which on a batch goes in two halves on two streams
  // of the batch whose kernels were launched last (a replayed graph launches none): did it go in halves, how was its last
  // part projected
  bool halved = false;
  kernels::project_shape projected;
  int64_t buffer_bytes  = 0;
  // what the arrays above are pieces of (see alloc): an allocation and its release take 0.6 ms of any size
  std::vector<dbuf> memory;
  size_t memory_used = 0;  // of the last of them
  // page-locked staging of calls with ordinary host memory, made when first needed: queries in,
  // results out (the last kernel of the batch writes them there)
  dbuf stage_q, stage_out;
  std::mutex mu;  // one search at a time per plan
  ~plan();
};

inline auto ix_debug(index_impl const& ix) -> debug_options { return ix.debug; }

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
                 bool wait     = false,
                 int max_lanes = 2);

/// True when a search with these device arrays works on them where they are (one process, everything in
/// the memory of the index's GPU, which is the current device); otherwise they are copied in and out.
auto search_in_place(index_impl const& ix, const float* queries, const int64_t* neighbors, const float* distances) -> bool;

/// One batch of the queries already on the GPU, launched kernel by kernel with an event between
/// them: milliseconds of center+sketch, projection, cell codes, lookup, first round, each wave,
/// best k (the per-kernel counterpart of detail::timed_batch, search.cu:965-981 of the reference).
auto profile_batch(resources const& res, search_params const& sp, index const& idx, int64_t nq,
                   int64_t k) -> std::vector<float>;

/// What the rounds of the plan's last batch looked like, six numbers for the first round and six for a wave
/// (zeros without one): threads of a block, blocks of a multiprocessor by shared memory, slots of the
/// gather's hash set, words of its bits (0: the set), 1 when the candidates are in global memory, 1 when the
/// fp16 rows leave the L2 cache first.
auto round_shapes(plan const& pl) -> std::vector<int32_t>;

/// The queries from which on a batch of the plan goes in two halves, 1 when the last one did, the form its projection took
/// (kernels::project_form) and the queries of a tile of it.
auto batch_forms(plan const& pl) -> std::vector<int32_t>;

/// Throws when a kernel of an earlier batch of this plan reported that it gave up (and clears the
/// report).
void check_tc(plan const& pl);

/// The batches of a call, dealt to its lanes in turn: run(lane, first row, rows) queues one, close(lane,
/// failed) is called once for every lane after the last, also when a batch could not be queued: what the
/// lanes hold by then runs all the same, and the next user of their plans has to come after it.
template <typename Run, typename Close>
void each_batch(int64_t nq, int m, int lanes, Run run, Close close)
{
  try {
    int64_t batch = 0;
    for (int64_t b0 = 0; b0 < nq; b0 += m, batch++)
      run(static_cast<int>(batch % lanes), b0, static_cast<int>(nq - b0 < m ? nq - b0 : m));
  } catch (...) {
    for (int l = 0; l < lanes; l++) {
      try {
        close(l, true);
      } catch (...) {  // the first error is the one to report
      }
    }
    throw;
  }
  for (int l = 0; l < lanes; l++)
    close(l, false);
}

/// The plan of these parameters for batches of up to m queries.
auto get_plan(index_impl& ix, search_params const& sp, int m, int k, int lane = 0) -> std::shared_ptr<plan>;

/// Bytes of one of the plan's arrays (`size` allocated) that belong to the last batch of m queries: a row
/// per query, `cap` rows allocated. With several processes the arrays hold this process's rows of a
/// batch, which is always a whole one.
inline auto bytes_used(int world, int cap, int m, size_t size) -> size_t
{
  return world > 1 ? size : size / static_cast<size_t>(cap > 0 ? cap : 1) * static_cast<size_t>(m);
}

}  // namespace octex_b200::detail
