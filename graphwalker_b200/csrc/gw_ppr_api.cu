// gw_ppr_api.cu -- C ABI of the multi-source PPR queries (gw_ppr_run,
// gw_ppr_autotune); the kernels are in gw_ppr.cu.
//
// The context's tables are not cleared between batches: each batch writes
// its slots under a new tag (QueryView::tag), which frees the slots of every
// earlier batch at once.  They are cleared when first allocated, when they
// grow, and when the tags run out (2^(32 - vertex id bits) - 1 of them: 63 at
// R-MAT scale 26).  GW_PPR_TAG_BITS caps the tag width (0 = untagged, every
// batch cleared), so that tests reach the wrap-around on small graphs.
//
// Tables are sized for the typical query (table_factor slots per walk of the
// budget).  A query whose table fills up is flagged by the kernel and run
// again, alone with the other flagged queries, with tables four times larger:
// its walks keep their stream ids, so the retried result is exactly the one a
// large enough table would have given.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "gw_ctx.h"
#include "gw_ppr.h"

namespace {

constexpr int kMaxRetries = 3;

uint64_t next_pow2(uint64_t x) {
  uint64_t p = 1;
  while (p < x) p <<= 1;
  return p;
}

// A set of queries laid out for one launch.  Everything a launch needs besides
// the tables lies in one staging range, written in pinned host memory and
// copied up at once, and everything it returns behind it, copied back at once:
// a query of a few hundred walks spent more time on fifteen small copies than
// on its walks.  Its device buffers are the context's (kept across calls) for
// the first round, its own for retries.
struct QuerySet {
  std::vector<uint32_t> qmap;  // index in the caller's query list
  std::vector<unsigned long long> prefix, id_base, toff;
  std::vector<uint32_t> sources, tmask;
  std::vector<unsigned long long> seg_first;  // top-k segments per query (prefix)
  std::vector<uint32_t> seg_slots;            // table slots of a segment: one for the set, or one per query
  uint64_t walks = 0, slots = 0;
  bool shared = false;        // the context's buffers (tagged), or this set's own (cleared, untagged)
  bool fresh_tables = false;  // d_tables was (re)allocated by upload_set: its content is undefined
  gw_devbuf own[3];
  gw_devbuf *d_stage, *d_tables, *d_cand;
  size_t back_at = 0, head_bytes = 0;  // the staging range: where the results start, and how much is copied up
  gw::QueryView qv{};
  unsigned long long* d_seg_first = nullptr;
  uint32_t *seg_done = nullptr, *seg_order = nullptr, *status = nullptr, *ids = nullptr, *cnt = nullptr;  // device

  QuerySet(gw_ctx* ctx, bool use_ctx_buffers) {
    gw_devbuf* b[3] = {&ctx->d_q_stage, &ctx->d_q_tables, &ctx->d_q_cand};
    gw_devbuf** d[3] = {&d_stage, &d_tables, &d_cand};
    for (int i = 0; i < 3; ++i) *d[i] = use_ctx_buffers ? b[i] : &own[i];
    shared = use_ctx_buffers;
  }
  ~QuerySet() {
    for (auto& b : own) b.release();
  }
};

// The results, as they lie behind the inputs: total visits, the status word
// (and padding), the table-full flags, then the lists.
struct Results {
  unsigned long long visits;
  uint32_t status, unused;
};
// Lists up to this size come back through the pinned staging; larger ones go
// straight to the caller's arrays.
constexpr size_t kStagedListBytes = 1u << 20;

gw_status plan_set(gw_ctx* ctx, const uint32_t* sources, const uint32_t* budgets, const unsigned long long* ids,
                   const std::vector<uint32_t>& which, uint64_t factor, QuerySet* s) {
  const uint32_t n = (uint32_t)which.size();
  s->qmap = which;
  s->sources.resize(n);
  s->prefix.assign(n + 1, 0);
  s->id_base.resize(n);
  s->toff.resize(n);
  s->tmask.resize(n);
  s->slots = 0;
  for (uint32_t i = 0; i < n; ++i) {
    const uint32_t q = which[i];
    if (sources[q] >= ctx->nv) return ctx->fail(GW_E_INVALID, "query %u: source %u >= nvertices", q, sources[q]);
    s->sources[i] = sources[q];
    s->prefix[i + 1] = s->prefix[i] + budgets[q];
    s->id_base[i] = ids[q];
    const uint64_t cap = next_pow2(std::max<uint64_t>(256, (uint64_t)budgets[q] * factor));
    if (cap > (1ull << 31)) return ctx->fail(GW_E_OVERFLOW, "query %u: visit table would exceed 2^31 slots", q);
    s->toff[i] = s->slots;
    s->tmask[i] = (uint32_t)(cap - 1);
    s->slots += cap;
  }
  s->walks = s->prefix[n];
  return GW_OK;
}

// batched: one launch ranks the whole set, and its segments go by all of it;
// one query at a time (plain), a launch ranks one, and its segments go by that
// query's table.
gw_status upload_set(gw_ctx* ctx, QuerySet* s, uint32_t k, cudaStream_t st, bool batched) {
  const size_t n = s->qmap.size();
  const void* tables0 = s->d_tables->p;
  const size_t table_bytes0 = s->d_tables->bytes;
  GW_CUDA(ctx, s->d_tables->ensure(s->slots * 8), "query tables alloc");
  s->fresh_tables = s->d_tables->p != tables0 || s->d_tables->bytes != table_bytes0;
  s->seg_first.resize(n + 1);
  if (batched) {
    s->seg_slots.assign(1, gw::topk_segment_slots(s->tmask.data(), (uint32_t)n, k));
    gw::topk_segment_prefix(s->tmask.data(), (uint32_t)n, s->seg_slots[0], s->seg_first.data());
  } else {
    s->seg_first[0] = 0;
    for (size_t q = 0; q < n; ++q) {
      s->seg_slots.push_back(gw::topk_segment_slots(&s->tmask[q], 1, k));
      unsigned long long one[2];
      gw::topk_segment_prefix(&s->tmask[q], 1, s->seg_slots[q], one);
      s->seg_first[q + 1] = s->seg_first[q] + one[1];
    }
  }
  const size_t nseg = s->seg_first[n];
  GW_CUDA(ctx, s->d_cand->ensure(nseg * k * 8 + 8), "top-k candidates");
  // 64-bit arrays first: prefix, seg_first (n + 1 each), id_base, toff, cursors
  // (n each); then sources, tmask, segment counters, segment order; then the results
  const size_t u64s = 2 * (n + 1) + 3 * n, u32s = 3 * n + nseg;
  s->back_at = (u64s * 8 + u32s * 4 + 7) / 8 * 8;
  s->head_bytes = s->back_at + sizeof(Results) + n * 4;
  GW_CUDA(ctx, s->d_stage->ensure(s->head_bytes + 2 * n * k * 4), "query alloc");
  GW_CUDA(ctx, ctx->h_q_stage.ensure(s->head_bytes + std::min(2 * n * k * 4, kStagedListBytes)), "query staging");
  char* const h = ctx->h_q_stage.as<char>();
  char* const d = s->d_stage->as<char>();
  memset(h, 0, s->head_bytes);  // cursors, segment counters, results start at zero
  size_t at = 0;
  auto put = [&](const void* src, size_t count, size_t width) {  // returns the array's place on the device
    if (src) memcpy(h + at, src, count * width);
    char* const where = d + at;
    at += count * width;
    return where;
  };
  s->qv.walk_prefix = reinterpret_cast<unsigned long long*>(put(s->prefix.data(), n + 1, 8));
  auto* seg_first = reinterpret_cast<unsigned long long*>(put(s->seg_first.data(), n + 1, 8));
  s->qv.id_base = reinterpret_cast<unsigned long long*>(put(s->id_base.data(), n, 8));
  s->qv.table_off = reinterpret_cast<unsigned long long*>(put(s->toff.data(), n, 8));
  s->qv.cursor = reinterpret_cast<unsigned long long*>(put(nullptr, n, 8));
  s->qv.sources = reinterpret_cast<uint32_t*>(put(s->sources.data(), n, 4));
  s->qv.table_mask = reinterpret_cast<uint32_t*>(put(s->tmask.data(), n, 4));
  s->seg_done = reinterpret_cast<uint32_t*>(put(nullptr, n, 4));
  s->seg_order = reinterpret_cast<uint32_t*>(d + at);
  if (batched)
    gw::topk_segment_order(s->tmask.data(), (uint32_t)n, s->seg_slots[0], s->seg_first.data(),
                           reinterpret_cast<uint32_t*>(h + at));
  Results* const r = reinterpret_cast<Results*>(d + s->back_at);
  s->qv.visits = &r->visits;
  s->status = &r->status;
  s->qv.full = reinterpret_cast<uint32_t*>(r + 1);
  s->ids = s->qv.full + n;
  s->cnt = s->ids + n * k;
  s->qv.tables = s->d_tables->as<unsigned long long>();
  s->qv.nq = (uint32_t)n;
  s->d_seg_first = seg_first;
  GW_CUDA(ctx, cudaMemcpyAsync(d, h, s->head_bytes, cudaMemcpyHostToDevice, st), "query copy");
  return GW_OK;
}

// Makes the set's tables free for a new batch: the next tag of the context's
// tables (cleared only when they are fresh or the tags have run out), or a
// clear of the set's own tables.  *cleared: a clear was launched.
cudaError_t assign_tag(gw_ctx* ctx, QuerySet* s, cudaStream_t st, bool* cleared) {
  *cleared = true;
  const uint32_t top = ctx->nv > 1 ? ctx->nv - 1 : 1;
  const uint32_t vbits = 32 - (uint32_t)__builtin_clz(top);  // bits of the largest vertex id
  uint32_t tbits = 32 - vbits;
  if (const char* cap = getenv("GW_PPR_TAG_BITS")) tbits = std::min<uint32_t>(tbits, (uint32_t)atoi(cap));
  const uint32_t ntags = tbits >= 2 ? (1u << tbits) - 1 : 0;  // the all-ones tag is the empty pattern's
  if (!s->shared || ntags == 0) {
    s->qv.tag = s->qv.tag_mask = 0;
    if (s->shared) ctx->q_tags_ok = false;  // untagged slots look like tag 0
    return gw::launch_clear_tables(s->qv.tables, s->slots, st);
  }
  cudaError_t e = cudaSuccess;
  if (s->fresh_tables || !ctx->q_tags_ok || ctx->q_tag_next >= ntags) {
    ctx->q_tags_ok = false;
    e = gw::launch_clear_tables(s->qv.tables, s->d_tables->bytes / 8, st);
    if (e != cudaSuccess) return e;
    ctx->q_tags_ok = true;
    ctx->q_tag_next = 0;
    s->fresh_tables = false;
  } else {
    *cleared = false;
  }
  s->qv.tag_mask = ~0u << vbits;
  s->qv.tag = ctx->q_tag_next++ << vbits;
  return e;
}

float elapsed(cudaEvent_t a, cudaEvent_t b) {
  float ms = 0.f;
  cudaEventElapsedTime(&ms, a, b);
  return ms;
}

// Tag (or clear) + walk + top-k of a whole set in two to four launches
// (batched), or clear + walk + top-k query by query (plain).  Timing events:
// ev[0] start, ev[1] tables free, ev[2] walked, ev[3] done.
cudaError_t run_set(gw_ctx* ctx, const gw_walk_params* p, const gw::WalkArgs& a, QuerySet* s, uint32_t k,
                    bool batched, int threads_per_sm, cudaStream_t st, cudaEvent_t* ev, uint32_t* launches) {
  cudaError_t e = cudaSuccess;
  const uint32_t n = s->qv.nq;
  cudaEventRecord(ev[0], st);
  bool cleared = false;
  e = assign_tag(ctx, s, st, &cleared);
  if (batched) {
    cudaEventRecord(ev[1], st);
    if (e == cudaSuccess)
      e = gw::launch_walk_queries((int)p->rule, s->qv, 0, s->walks, ctx->view(), a, s->status, threads_per_sm, st);
    cudaEventRecord(ev[2], st);
    if (e == cudaSuccess)
      e = gw::launch_topk_segmented(s->qv, 0, n, k, s->ids, s->cnt, s->d_seg_first, s->seg_first.data(),
                                    s->seg_slots[0], s->d_cand->as<unsigned long long>(), s->seg_done, s->seg_order, st);
    cudaEventRecord(ev[3], st);
    *launches += (s->seg_first[n] > n && !gw::topk_is_few(s->seg_first.data(), n, s->seg_slots[0], k) ? 3 : 2) + (cleared ? 1 : 0);
  } else {
    cudaEventRecord(ev[1], st);
    *launches += cleared ? 1 : 0;
    for (uint32_t q = 0; q < n && e == cudaSuccess; ++q) {
      e = gw::launch_clear_tables(s->qv.tables + s->toff[q], (uint64_t)s->tmask[q] + 1, st);
      gw::QueryView one = s->qv;
      one.cursor += q;
      if (e == cudaSuccess)
        e = gw::launch_walk_queries((int)p->rule, one, s->prefix[q], s->prefix[q + 1], ctx->view(), a, s->status, 0, st);
      if (e == cudaSuccess)
        e = gw::launch_topk_segmented(s->qv, q, 1, k, s->ids, s->cnt, s->d_seg_first, s->seg_first.data(),
                                      s->seg_slots[q], s->d_cand->as<unsigned long long>(), s->seg_done, nullptr, st);
      if (s->seg_first[q + 1] - s->seg_first[q] > 1 && !gw::topk_is_few(&s->seg_first[q], 1, s->seg_slots[q], k)) ++*launches;
    }
    cudaEventRecord(ev[2], st);
    cudaEventRecord(ev[3], st);
    *launches += 3 * n;
  }
  return e;
}

}  // namespace

extern "C" gw_status gw_ppr_run(gw_ctx* ctx, const gw_walk_params* params, const uint32_t* sources,
                                const uint32_t* budgets, uint32_t nq, uint32_t k, uint32_t batched,
                                uint32_t* topk_ids, uint32_t* topk_counts, gw_ppr_stats* stats) {
  if (!ctx) return GW_E_INVALID;
  if (ctx->residency != GW_RESIDENT_HBM) return ctx->fail(GW_E_STATE, "PPR queries need a resident graph");
  if (nq == 0) return GW_OK;
  if (!sources || !budgets || !topk_ids || !topk_counts) return ctx->fail(GW_E_INVALID, "NULL buffer");
  if (k == 0 || k > gw::kTopkMaxK) return ctx->fail(GW_E_INVALID, "k must lie in [1, %u]", gw::kTopkMaxK);
  gw::WalkArgs a;
  gw_status s = gw::make_walk_args(ctx, params, &a);
  if (s != GW_OK) return s;
  // stream id of each query's first walk: budgets laid end to end
  std::vector<unsigned long long> ids(nq);
  unsigned long long total = 0;
  for (uint32_t q = 0; q < nq; ++q) {
    ids[q] = total;
    total += budgets[q];
  }
  std::vector<uint32_t> which(nq);
  for (uint32_t q = 0; q < nq; ++q) which[q] = q;
  uint64_t factor = params->table_factor ? params->table_factor : 8;
  cudaStream_t st = ctx->stream;
  cudaEvent_t* const ev = ctx->q_events;
  for (int i = 0; i < 4; ++i)
    if (!ev[i]) GW_CUDA(ctx, cudaEventCreate(&ev[i]), "event");
  gw_ppr_stats local{};
  local.walks = total;
  std::vector<uint32_t> lists;
  for (int round = 0; round <= kMaxRetries && !which.empty(); ++round) {
    QuerySet set(ctx, round == 0);
    s = plan_set(ctx, sources, budgets, ids.data(), which, factor, &set);
    const bool b = batched || round > 0;
    if (s == GW_OK) s = upload_set(ctx, &set, k, st, b);
    if (s != GW_OK) break;
    set.qv.chunk = ctx->ppr_chunk;
    cudaError_t e = run_set(ctx, params, a, &set, k, b, b ? ctx->ppr_threads_per_sm : 0, st, ev, &local.launches);
    const uint32_t n = (uint32_t)which.size();
    const size_t nk = (size_t)n * k;
    // The first round holds every query in the caller's order: long lists go
    // straight into the caller's arrays (a rerun query's rows are overwritten
    // later); short ones and a rerun's go through host memory to their rows.
    const bool staged = 2 * nk * 4 <= kStagedListBytes, direct = round == 0 && !staged;
    char* const back = ctx->h_q_stage.as<char>() + set.back_at;
    const size_t head = sizeof(Results) + (size_t)n * 4;
    uint32_t* hid = topk_ids;
    uint32_t* hcnt = topk_counts;
    if (staged) {
      hid = reinterpret_cast<uint32_t*>(back + head);
      hcnt = hid + nk;
    } else if (!direct) {
      lists.resize(2 * nk);
      hid = lists.data();
      hcnt = hid + nk;
    }
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(back, set.d_stage->as<char>() + set.back_at, head + (staged ? 2 * nk * 4 : 0),
                          cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess && !staged) e = cudaMemcpyAsync(hid, set.ids, nk * 4, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess && !staged) e = cudaMemcpyAsync(hcnt, set.cnt, nk * 4, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
      s = ctx->cuda_fail(e, "gw_ppr_run");
      break;
    }
    const Results* const res = reinterpret_cast<const Results*>(back);
    const uint32_t* const full = reinterpret_cast<const uint32_t*>(res + 1);
    local.visits += res->visits;
    s = gw::status_of(ctx, res->status);
    if (s != GW_OK) break;
    if (round == 0 && b) {
      local.ms_clear = elapsed(ev[0], ev[1]);
      local.ms_walk = elapsed(ev[1], ev[2]);
      local.ms_topk = elapsed(ev[2], ev[3]);
    }
    local.ms_total += elapsed(ev[0], ev[3]);
    local.table_slots += set.slots;
    std::vector<uint32_t> again;
    for (uint32_t i = 0; i < n; ++i) {
      const uint32_t q = which[i];
      if (full[i]) {
        again.push_back(q);
        continue;
      }
      if (direct) continue;
      std::copy(hid + (size_t)i * k, hid + (size_t)(i + 1) * k, topk_ids + (size_t)q * k);
      std::copy(hcnt + (size_t)i * k, hcnt + (size_t)(i + 1) * k, topk_counts + (size_t)q * k);
    }
    which.swap(again);
    factor *= 4;
  }
  if (s == GW_OK && !which.empty())
    s = ctx->fail(GW_E_OVERFLOW, "%zu queries still filled their visit tables after %d retries",
                  which.size(), kMaxRetries);
  if (s != GW_OK) {
    // The queries without a complete list (still in `which`) get empty rows
    // (ids all-ones, counts 0), so a partial round-0 list is never mistaken
    // for a result.  Copies into those rows may still be queued: wait first.
    cudaStreamSynchronize(st);
    for (const uint32_t q : which) {
      std::fill(topk_ids + (size_t)q * k, topk_ids + (size_t)(q + 1) * k, 0xffffffffu);
      std::fill(topk_counts + (size_t)q * k, topk_counts + (size_t)(q + 1) * k, 0u);
    }
  }
  if (stats) *stats = local;
  return s;
}

extern "C" gw_status gw_ppr_autotune(gw_ctx* ctx, const gw_walk_params* params, const uint32_t* sources,
                                     const uint32_t* budgets, uint32_t nq, uint32_t* threads_per_sm,
                                     uint32_t* walks_per_chunk) {
  if (!ctx) return GW_E_INVALID;
  if (nq == 0 || !sources || !budgets) return ctx->fail(GW_E_INVALID, "empty sample");
  gw::WalkArgs a;
  gw_status s = gw::make_walk_args(ctx, params, &a);
  if (s != GW_OK) return s;
  std::vector<unsigned long long> ids(nq);
  unsigned long long total = 0;
  for (uint32_t q = 0; q < nq; ++q) {
    ids[q] = total;
    total += budgets[q];
  }
  std::vector<uint32_t> which(nq);
  for (uint32_t q = 0; q < nq; ++q) which[q] = q;
  QuerySet set(ctx, true);
  s = plan_set(ctx, sources, budgets, ids.data(), which, params->table_factor ? params->table_factor : 8, &set);
  if (s == GW_OK) s = upload_set(ctx, &set, 1, ctx->stream, true);
  if (s != GW_OK) return s;
  cudaStream_t st = ctx->stream;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  // launch shape (threads per SM) x walks per cursor grab
  const int thread_candidates[] = {512, 1024, 1536, 2048};
  const uint32_t chunk_candidates[] = {64, 128, 256, 512};
  int best = 0;
  uint32_t best_chunk = gw::kWarpChunk;
  float best_ms = 1e30f;
  for (int c : thread_candidates) {
    for (uint32_t ch : chunk_candidates) {
      set.qv.chunk = ch;
      float ms_sum = 0.f;
      for (int rep = 0; rep < 3; ++rep) {
        bool cleared = false;
        if (assign_tag(ctx, &set, st, &cleared) != cudaSuccess) break;
        cudaMemsetAsync(set.qv.cursor, 0, sizeof(unsigned long long), st);
        cudaEventRecord(e0, st);
        gw::launch_walk_queries((int)params->rule, set.qv, 0, set.walks, ctx->view(), a,
                                ctx->d_status.as<uint32_t>(), c, st);
        cudaEventRecord(e1, st);
        cudaEventSynchronize(e1);
        if (rep) ms_sum += elapsed(e0, e1);  // the first run warms up
      }
      if (ms_sum < best_ms) {
        best_ms = ms_sum;
        best = c;
        best_chunk = ch;
      }
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  s = gw::take_status(ctx, st);
  if (s != GW_OK) return s;
  ctx->ppr_threads_per_sm = best;
  ctx->ppr_chunk = best_chunk;
  if (threads_per_sm) *threads_per_sm = (uint32_t)best;
  if (walks_per_chunk) *walks_per_chunk = best_chunk;
  return GW_OK;
}
