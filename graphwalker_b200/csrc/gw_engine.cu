// gw_engine.cu -- GraphWalker's block loop on the device.
//
//   graphwalker_engine::run            src/engine/graphwalker.hpp:272-311
//   findSubGraph / loadSubGraph        src/engine/graphwalker.hpp:168-234
//   swapOut (evict fewest walks)       src/engine/graphwalker.hpp:236-251
//   WalkManager::chooseBlock & co.     src/walks/walk.hpp:204-252
//   getCurrentWalks / updateWalkNum    src/walks/walk.hpp:114-192
//   writeWalks2Disk / readWalksfromDisk src/walks/walk.hpp:103-157 (pool budget)
//
// Each superstep picks a block with the reference's state-aware policy (with
// probability `prob` the block holding the lowest-hop walk, otherwise the
// block with the most pending walks), makes its CSR available (resident HBM,
// or a slot filled from pinned host memory by async copies on a side stream),
// advances every walk of its pool while it stays inside the block, and stably
// partitions the walks that left into the pools of their new blocks.  The
// three kernels of a superstep (walk, scan, scatter) are queued together: the
// device keeps the table of pools, so the scatter needs nothing from the
// host, and the pending counts and minimum hops the policy reads reach the
// host through mapped pinned memory as soon as the scan is done, while the
// scatter runs.  Only a superstep that outgrows a pool waits for the host.
// (At R-MAT scale 22 with 33 blocks and 4.2 M walks, 299 supersteps: 64 us a
// superstep with five partition launches and a synchronisation before the
// scatter; see gw_partition.cu.)
//
// Streaming differs from findSubGraph in three ways that change neither the
// order of blocks nor any walk:
//  * the row pointer stays in HBM, and a slot holds a block's column slice;
//  * a chosen block in no slot whose pool is small (ctx->mapped_max_walks,
//    or per block its column bytes / kMappedBytesPerWalk) is read in place
//    from the pinned host columns through their mapped device address: each
//    hop fetches one sector over the host link instead of the whole block;
//  * while a block runs, up to kCopyAhead blocks with many pending walks are
//    copied into slots before their turn, each taking the room of the slot
//    with the fewest pending walks (swapOut's victim) when it has more.
//
// With a pool budget (ctx->pool_budget), walk pools beyond it wait in a
// pinned host arena, in either residency; a pool is the arena part (older
// walks) followed by its device part, so pool order is kept.
#include <algorithm>
#include <cstring>

#include "gw_ctx.h"

namespace gw {

namespace {

constexpr uint32_t kNoBlock = 0xffffffffu;
// GW_MAPPED_AUTO: a streamed block runs in place when it has at most one
// pending walk per this many bytes of its column slice.  Copying a block
// costs its bytes at the host link's rate; a walk run in place costs a sector
// per hop fetched over the same link and waits on its latency.
constexpr uint64_t kMappedBytesPerWalk = 128;
// Blocks copied ahead of their turn at most (1 to 5 measured within 2 % of
// one another on an out-of-core scale-27 graph, the deeper the faster).
constexpr size_t kCopyAhead = 3;

// chooseBlock (walk.hpp:245-252) over the engine's pending counts.
uint32_t block_with_max_walks(const std::vector<uint64_t>& walknum) {
  uint64_t maxw = 0;
  uint32_t maxp = 0;
  for (uint32_t p = 0; p < walknum.size(); ++p)
    if (maxw < walknum[p]) {
      maxw = walknum[p];
      maxp = p;
    }
  return maxp;
}

uint32_t block_with_min_step(const std::vector<uint64_t>& walknum, const std::vector<uint32_t>& minstep) {
  uint32_t mins = 0xffff, minp = 0;
  for (uint32_t p = 0; p < minstep.size(); ++p)
    if (mins > minstep[p]) {
      mins = minstep[p];
      minp = p;
    }
  if (walknum[minp] > 0) return minp;
  return block_with_max_walks(walknum);
}

uint32_t choose_block(const std::vector<uint64_t>& walknum, const std::vector<uint32_t>& minstep,
                      float prob, uint64_t seed, uint64_t superstep) {
  // the reference's coin is ((float)rand())/RAND_MAX; here its 31-bit draw
  // comes from Philox(seed, (superstep, "CHOS")) so a run is reproducible
  const Philox4 ph = philox4x32_10((uint32_t)superstep, (uint32_t)(superstep >> 32), 0x43484F53u,
                                   0u, (uint32_t)seed, (uint32_t)(seed >> 32));
  const float cc = (float)(int32_t)(ph.x >> 1) / 2147483647;
  if (cc < prob) return block_with_min_step(walknum, minstep);
  return block_with_max_walks(walknum);
}

}  // namespace

gw_status run_blocked(gw_ctx* ctx, const gw_walk_params* p) {
  WalkArgs a;
  gw_status s = make_walk_args(ctx, p, &a);
  if (s != GW_OK) return s;
  if (p->sink == GW_SINK_PATH_RECORD)
    return ctx->fail(GW_E_INVALID, "PATH_RECORD needs GW_MODE_RESIDENT");
  const uint32_t nb = ctx->nblocks;
  if (nb >= kMaxBuckets) return ctx->fail(GW_E_INVALID, "at most 7999 blocks in blocked mode");
  // Owned blocks (one rank of a vertex-partitioned run): only the blocks in
  // [own_lo, own_hi) execute, and walks that move to other blocks wait in
  // those blocks' pools for gw_read_pool.  block_hi = 0: every block.
  const uint32_t own_lo = p->block_hi ? p->block_lo : 0, own_hi = p->block_hi ? p->block_hi : nb;
  if (own_lo >= own_hi || own_hi > nb)
    return ctx->fail(GW_E_INVALID, "owned blocks [%u, %u) not inside [0, %u)", p->block_lo, p->block_hi, nb);
  const bool restricted = own_lo > 0 || own_hi < nb;
  const bool streaming = ctx->residency == GW_STREAM_PINNED;
  cudaStream_t st = ctx->stream, xs = ctx->copy_stream;

  // ---- initial pools (startWalks; getCurrentWalks reads them back) ----
  ctx->pools.resize(nb);
  ctx->pool_chunks.assign(nb, {});
  ctx->pool_host_n.assign(nb, 0);
  ctx->pool_size.assign(nb, 0);
  ctx->minstep.assign(nb, 0xffff);
  ctx->stats = gw_run_stats{};
  // What the run needs besides its pools comes first.  Where it does not fit
  // beside the pools an earlier run left, those go back: their walks are gone,
  // and in parts of one slab they may hold more than this run will.
  auto ensure = [&](gw_devbuf& b, size_t bytes) -> cudaError_t {
    cudaError_t e = b.ensure(bytes);
    if (e != cudaErrorMemoryAllocation || !ctx->pool_slab.p) return e;
    cudaGetLastError();
    ctx->release_pools();
    return b.ensure(bytes);
  };
  uint64_t all = 0, maxpool = 0;
  for (uint32_t b = 0; b < nb; ++b) {
    all += ctx->pool_words[b].size();
    maxpool = std::max<uint64_t>(maxpool, ctx->pool_words[b].size());
  }
  GW_CUDA(ctx, ensure(ctx->d_words, maxpool * 8), "word alloc");
  if (ctx->pools_have_ids) GW_CUDA(ctx, ensure(ctx->d_ids, maxpool * 4), "id alloc");

  // ---- sinks ----
  SinkView sv{};
  GW_CUDA(ctx, ensure(ctx->d_counts, (size_t)ctx->nv * 4), "counts alloc");
  GW_CUDA(ctx, cudaMemsetAsync(ctx->d_counts.p, 0, (size_t)ctx->nv * 4, st), "counts clear");
  GW_CUDA(ctx, ensure(ctx->d_closure, 8), "closure alloc");
  GW_CUDA(ctx, cudaMemsetAsync(ctx->d_closure.p, 0, 8, st), "closure clear");
  sv.counts = ctx->d_counts.as<uint32_t>();
  sv.closure = ctx->d_closure.as<unsigned long long>();

  // ---- streamed block slots ----
  // One device slot holds the column slice of one block,
  //   csr[beg_pos[blocks[b]] .. beg_pos[blocks[b+1]]);
  // the row pointer of every block stays in HBM.
  auto& slots = ctx->slots;
  std::vector<uint32_t> slot_block;  // block held, kNoBlock if empty
  std::vector<int> slot_of;          // per block: slot index or -1
  const uint32_t nslots = streaming ? std::max<uint32_t>(2, std::min(ctx->nmblocks, nb)) : 0;
  uint64_t max_e = 0;
  if (streaming) {
    const uint64_t* hr = ctx->h_rowptr.as<uint64_t>();
    for (uint32_t b = 0; b < nb; ++b) max_e = std::max<uint64_t>(max_e, hr[ctx->blocks[b + 1]] - hr[ctx->blocks[b]]);
  }
  struct SlotRelease {  // large slots go back to the device when the run ends
    gw_ctx* ctx;
    bool drop;
    ~SlotRelease() {
      if (!drop) return;
      cudaStreamSynchronize(ctx->copy_stream);
      cudaStreamSynchronize(ctx->stream);
      ctx->slots.release();
    }
  } slot_release{ctx, streaming && nslots * max_e * 4 > gw_ctx::BlockSlots::kKeptSlotBytes};
  if (streaming) {
    slot_block.assign(nslots, kNoBlock);
    slot_of.assign(nb, -1);
    if (slots.csr.size() != nslots) slots.release();
    slots.csr.resize(nslots);
    while (slots.ready.size() < nslots) {
      cudaEvent_t ev[2] = {};
      for (auto& x : ev) GW_CUDA(ctx, cudaEventCreateWithFlags(&x, cudaEventDisableTiming), "slot event");
      slots.ready.push_back(ev[0]);
      slots.free_ev.push_back(ev[1]);
    }
    for (uint32_t i = 0; i < nslots; ++i) {
      GW_CUDA(ctx, ensure(slots.csr[i], std::max<uint64_t>(max_e, 1) * 4), "slot alloc");
      cudaEventRecord(slots.free_ev[i], st);
    }
  }
  // Without a budget the pools start as parts of one allocation: one
  // allocation instead of one per block.  A part holds its walks, or what its
  // pool held after an earlier run; and, so that few pools must grow, an even
  // share of all walks more, where the device has room for that whatever the
  // walks do: every pool growing, one after the other, until it could hold all
  // of them (twice over, and one being copied).  Elsewhere, as on a device
  // that the streamed graph's slots fill, the pools take no more than each by
  // itself would.  Pools that an earlier run grew past their parts leave those
  // idle, so they are laid out anew.  (A budget moves pools out one by one, so
  // each is then its own.)
  {
    bool fits = true, idle = false;
    std::vector<uint64_t> room(nb), roomy(nb);
    uint64_t want = 0, want_roomy = 0;
    for (uint32_t b = 0; b < nb; ++b) {
      const uint64_t m = ctx->pool_words[b].size(), held = ctx->pools[b].bytes / sizeof(gw_walk_rec);
      fits = fits && held >= m;
      idle = idle || (ctx->pool_slab.p && ctx->pools[b].p && !ctx->in_slab(ctx->pools[b].p));
      room[b] = std::max(held, m);
      roomy[b] = std::max<uint64_t>(held, m + all / nb + 1024);
      want += room[b];
      want_roomy += roomy[b];
    }
    if (ctx->pool_budget) {
      if (ctx->pool_slab.p) ctx->release_pools();
    } else if (!fits || idle) {
      ctx->release_pools();
      const uint64_t most = std::max<uint64_t>(2 * all, 1024);  // what a pool may grow to
      size_t free_bytes = 0, total_bytes = 0;
      GW_CUDA(ctx, cudaMemGetInfo(&free_bytes, &total_bytes), "free memory");
      // beside the pools: 4 bytes a walk of destinations, grown by halves, and the tile counts
      const double needed = (double)sizeof(gw_walk_rec) * (want_roomy + (double)(nb + 1) * most) + 16.0 * all +
                            (double)nb * 4 * (1184 + all / (kMaxRows * (uint64_t)kWalkThreads));
      if (needed <= (double)free_bytes) {
        room.swap(roomy);
        want = want_roomy;
      }
      if (want && ctx->pool_slab.ensure(want * sizeof(gw_walk_rec)) == cudaSuccess) {
        uint64_t at = 0;
        for (uint32_t b = 0; b < nb; ++b) {
          if (!room[b]) continue;
          ctx->pools[b].p = ctx->pool_slab.as<gw_walk_rec>() + at;
          ctx->pools[b].bytes = room[b] * sizeof(gw_walk_rec);
          at += room[b];
        }
      } else {
        cudaGetLastError();  // no room for all at once: each pool by itself, below
      }
    }
  }
  std::vector<uint64_t> cap(nb, 0);
  for (uint32_t b = 0; b < nb; ++b) cap[b] = ctx->pools[b].bytes / sizeof(gw_walk_rec);
  // Grown pools come from the stream-ordered allocator, so replacing one
  // queues its free behind the copy out of it; a pool from an earlier run is
  // retired instead and freed with the events, and a part of the slab stays
  // with the slab.
  std::vector<char> pool_async(nb, 0);
  auto retire = [&](uint32_t d, std::vector<void*>* retired) {
    if (!ctx->pools[d].p || ctx->in_slab(ctx->pools[d].p)) return;
    if (pool_async[d]) cudaFreeAsync(ctx->pools[d].p, st);
    else retired->push_back(ctx->pools[d].p);
  };
  // records of block d's pool held on the device (after its host part)
  auto dev_n = [&](uint32_t d) { return ctx->pool_size[d] - ctx->pool_host_n[d]; };
  constexpr uint64_t kChunk = gw_ctx::kPoolChunk;
  if (ctx->pool_budget) {
    // pinned chunks for every walk of the run, plus a partly filled one per block
    const uint64_t nchunks = (all + kChunk - 1) / kChunk + nb;
    GW_CUDA(ctx, ctx->pool_arena.ensure(nchunks * kChunk * sizeof(gw_walk_rec)), "pool arena");
    ctx->arena_free.resize(nchunks);
    for (uint64_t c = 0; c < nchunks; ++c) ctx->arena_free[c] = (uint32_t)(nchunks - 1 - c);
  }
  gw_walk_rec* const arena = ctx->pool_arena.as<gw_walk_rec>();
  // writeWalks2Disk: once the device pools hold more than the budget, the
  // pools with the fewest pending walks (never the fullest) move to host
  // memory, empty pools first giving back their room, until they hold half
  // of it: the headroom takes many supersteps' arrivals before the next
  // spill, so pools move out in a few large batches, not a few every step.
  auto spill_to_budget = [&](bool* moved) -> cudaError_t {
    if (!ctx->pool_budget) return cudaSuccess;
    uint64_t held = 0;
    for (uint32_t d = 0; d < nb; ++d) held += cap[d];
    if (held * sizeof(gw_walk_rec) <= ctx->pool_budget) return cudaSuccess;
    *moved = true;
    const uint64_t low = ctx->pool_budget / 2;
    uint32_t fullest = 0;
    for (uint32_t d = 1; d < nb; ++d)
      if (ctx->pool_size[d] > ctx->pool_size[fullest]) fullest = d;
    std::vector<uint32_t> order;
    for (uint32_t d = 0; d < nb; ++d)
      if (cap[d] && d != fullest) order.push_back(d);
    std::stable_sort(order.begin(), order.end(), [&](uint32_t x, uint32_t y) {
      const bool ex = dev_n(x) == 0, ey = dev_n(y) == 0;
      return ex != ey ? ex : ctx->pool_size[x] < ctx->pool_size[y];
    });
    // Copies out and frees of stream-ordered pools queue on st behind the
    // scatter that filled them; pools from gw_walks_add are freed after a
    // synchronisation.
    cudaError_t e = cudaSuccess;
    std::vector<void*> sync_free;
    for (size_t i = 0; i < order.size() && e == cudaSuccess && held * sizeof(gw_walk_rec) > low; ++i) {
      const uint32_t d = order[i];
      const uint64_t dn = dev_n(d);
      for (uint64_t off = 0; off < dn && e == cudaSuccess;) {
        uint64_t& hn = ctx->pool_host_n[d];
        const uint64_t used = hn % kChunk;
        if (used == 0) {
          if (ctx->arena_free.empty()) return cudaErrorMemoryAllocation;
          ctx->pool_chunks[d].push_back(ctx->arena_free.back());
          ctx->arena_free.pop_back();
        }
        const uint64_t c = ctx->pool_chunks[d].back(), m = std::min(kChunk - used, dn - off);
        e = cudaMemcpyAsync(arena + c * kChunk + used, ctx->pools[d].as<gw_walk_rec>() + off,
                            m * sizeof(gw_walk_rec), cudaMemcpyDeviceToHost, st);
        hn += m;
        off += m;
      }
      if (e != cudaSuccess) break;
      if (dn) ctx->stats.pools_spilled++;
      if (pool_async[d]) e = cudaFreeAsync(ctx->pools[d].p, st);
      else sync_free.push_back(ctx->pools[d].p);
      ctx->pools[d].p = nullptr;
      ctx->pools[d].bytes = 0;
      held -= cap[d];
      cap[d] = 0;
      pool_async[d] = 0;
    }
    if (!sync_free.empty()) {
      const cudaError_t e2 = cudaStreamSynchronize(st);
      for (void* q : sync_free) cudaFree(q);
      if (e == cudaSuccess) e = e2;
    }
    return e;
  };
  uint64_t walksum = 0;
  // Mapped pinned memory the host and a superstep's kernels share, reached by
  // the device at its mapped address, so the small transfers of a superstep
  // never wait behind a block copy on the copy engine: what the scan reports
  // per block (moved_word), and two copies of the pool table (one for the next
  // superstep's launch, one for pools grown in the middle of a superstep: each
  // is read by a kernel the host has waited for before it writes that copy
  // again).
  GW_CUDA(ctx, ctx->h_xfer.ensure(9 * (size_t)nb * 8), "pinned scratch");
  volatile uint64_t* const h_moved = ctx->h_xfer.as<uint64_t>();
  uint64_t* const h_table = ctx->h_xfer.as<uint64_t>() + nb;
  void* m_xfer = nullptr;
  GW_CUDA(ctx, cudaHostGetDevicePointer(&m_xfer, ctx->h_xfer.p, 0), "mapped scratch");
  uint64_t* const m_moved = static_cast<uint64_t*>(m_xfer);
  const uint64_t* const m_table = m_moved + nb;
  std::vector<uint32_t> h_minhop(nb), h_totals(nb);
  // device: minimum hops (reset by each scan after it has read them; the
  // initial pools' lie behind them, side by side), the pool table, and the
  // superstep clock
  const size_t minhop_words = (size_t)nb * (kMinhopStride + 1);
  GW_CUDA(ctx, ctx->d_minhop.ensure(minhop_words * 4), "minhop alloc");
  GW_CUDA(ctx, cudaMemsetAsync(ctx->d_minhop.p, 0xff, minhop_words * 4, st), "minhop clear");
  uint32_t* const pool_minhop = ctx->d_minhop.as<uint32_t>() + (size_t)nb * kMinhopStride;
  const size_t entries = PoolTable::stride(nb), table_bytes = 4 * entries * 8 + 8 + kClockWords * 8;
  GW_CUDA(ctx, ctx->d_pool_table.ensure(table_bytes), "pool table alloc");
  GW_CUDA(ctx, cudaMemsetAsync(ctx->d_pool_table.p, 0, table_bytes, st), "pool table clear");
  PoolTable table;
  table.ptr = ctx->d_pool_table.as<gw_walk_rec*>();
  table.n = ctx->d_pool_table.as<uint64_t>() + entries;
  table.cap = table.n + entries;
  table.place = table.cap + entries;
  table.full = reinterpret_cast<uint32_t*>(table.place + entries);
  PartitionScratch ps{};
  ps.minhop = ctx->d_minhop.as<uint32_t>();
  ps.clock = reinterpret_cast<unsigned long long*>(table.full + 2);
  for (uint32_t b = 0; b < nb; ++b) {
    const uint64_t m = ctx->pool_words[b].size();
    if (!m) continue;
    if (cap[b] < m) {
      GW_CUDA(ctx, ctx->pools[b].ensure(m * sizeof(gw_walk_rec)), "pool alloc");
      cap[b] = m;
    }
    GW_CUDA(ctx, cudaMemcpyAsync(ctx->d_words.p, ctx->pool_words[b].data(), m * 8,
                                 cudaMemcpyHostToDevice, st), "walk upload");
    if (ctx->pools_have_ids)
      GW_CUDA(ctx, cudaMemcpyAsync(ctx->d_ids.p, ctx->pool_ids[b].data(), m * 4,
                                   cudaMemcpyHostToDevice, st), "id upload");
    GW_CUDA(ctx, launch_unpack_words(ctx->d_words.as<uint64_t>(),
                                     ctx->pools_have_ids ? ctx->d_ids.as<uint32_t>() : nullptr, m,
                                     ctx->blocks[b], ctx->pools[b].as<gw_walk_rec>(), st, pool_minhop + b), "unpack");
    ctx->pool_size[b] = m;
    walksum += m;
    bool moved = false;
    GW_CUDA(ctx, spill_to_budget(&moved), "pool spill");
  }
  GW_CUDA(ctx, cudaMemcpyAsync(h_minhop.data(), pool_minhop, (size_t)nb * 4, cudaMemcpyDeviceToHost, st), "minimum hops");
  GW_CUDA(ctx, cudaStreamSynchronize(st), "walk upload");
  for (uint32_t b = 0; b < nb; ++b) {
    ctx->minstep[b] = std::min<uint32_t>(h_minhop[b], 0xffffu);
    h_moved[b] = 0;
  }
  const uint64_t nwalks = walksum;
  walksum = 0;  // from here on: walks pending in the owned blocks
  for (uint32_t b = own_lo; b < own_hi; ++b) walksum += ctx->pool_size[b];
  std::vector<uint64_t> own_num;
  std::vector<uint32_t> own_min;

  // mapped device address of the pinned host columns (blocks read in place)
  const uint32_t* m_colidx = nullptr;
  if (streaming && ctx->mapped_max_walks) {
    void* mp = nullptr;
    const cudaError_t me = cudaHostGetDevicePointer(&mp, ctx->h_colidx.p, 0);
    if (me == cudaSuccess) {
      m_colidx = static_cast<const uint32_t*>(mp);
    } else if (ctx->mapped_max_walks == GW_MAPPED_AUTO) {
      cudaGetLastError();  // no mapped host memory here: the default copies every block
    } else {
      return ctx->cuda_fail(me, "mapped colidx (gw_set_mapped_block_walks)");
    }
  }
  // the most pending walks at which block q runs in place (0 = never)
  auto mapped_limit = [&](uint32_t q) -> uint64_t {
    if (!m_colidx) return 0;
    if (ctx->mapped_max_walks != GW_MAPPED_AUTO) return ctx->mapped_max_walks;
    const uint64_t* hr = ctx->h_rowptr.as<uint64_t>();
    return (hr[ctx->blocks[q + 1]] - hr[ctx->blocks[q]]) * 4 / kMappedBytesPerWalk;
  };
  ctx->stats.walks = nwalks;

  std::vector<uint32_t> ahead;  // blocks copied ahead of their turn, not yet run
  // findSubGraph: make block b resident in a slot (never the slot `keep`).
  auto load_block = [&](uint32_t b, int keep) -> int {
    if (slot_of[b] >= 0) return slot_of[b];
    int victim = -1;
    for (uint32_t i = 0; i < nslots && victim < 0; ++i)
      if (slot_block[i] == kNoBlock && (int)i != keep) victim = (int)i;
    if (victim < 0) {  // swapOut: resident block with the fewest pending walks
      uint64_t minw = ~0ull;
      for (uint32_t i = 0; i < nslots; ++i) {
        if ((int)i == keep) continue;
        const uint64_t w = ctx->pool_size[slot_block[i]];
        if (w < minw) {
          minw = w;
          victim = (int)i;
        }
      }
      slot_of[slot_block[victim]] = -1;
      ahead.erase(std::remove(ahead.begin(), ahead.end(), slot_block[victim]), ahead.end());
    }
    const uint64_t* hr = ctx->h_rowptr.as<uint64_t>();
    const uint32_t v0 = ctx->blocks[b], v1 = ctx->blocks[b + 1];
    const uint64_t e0 = hr[v0], e1 = hr[v1];
    cudaStreamWaitEvent(xs, slots.free_ev[victim], 0);
    if (e1 > e0)
      cudaMemcpyAsync(slots.csr[victim].p, ctx->h_colidx.as<uint32_t>() + e0, (e1 - e0) * 4,
                      cudaMemcpyHostToDevice, xs);
    cudaEventRecord(slots.ready[victim], xs);
    slot_block[victim] = b;
    slot_of[b] = victim;
    ctx->stats.block_loads++;
    ctx->stats.bytes_h2d += (e1 - e0) * 4;
    return victim;
  };

  double ms_copy_wait = 0;
  // run start/end, and a superstep's wait for a block copy.  Destroyed on
  // every return; so are the pools that grown pools replaced, once no queued
  // copy reads them.
  struct Events {
    cudaEvent_t e[4];
    std::vector<void*> retired;
    Events() {
      for (auto& x : e) cudaEventCreate(&x);
    }
    ~Events() {
      for (auto& x : e) cudaEventDestroy(x);
      for (void* p : retired) cudaFree(p);
    }
  } evs;
  cudaEvent_t t0 = evs.e[0], t1 = evs.e[1];
  // The device's pool table from the host's, by a kernel on st: `at` is the
  // copy in mapped memory (0: before a superstep, 1: pools grown inside one),
  // `arrived` the walks the queued scatter adds to each pool (NULL: none).
  auto upload_table = [&](int at, const uint32_t* arrived) {
    uint64_t* t = h_table + (size_t)at * 4 * nb;
    for (uint32_t d = 0; d < nb; ++d) {
      t[d] = reinterpret_cast<uint64_t>(ctx->pools[d].p);
      t[nb + d] = dev_n(d) + (arrived ? arrived[d] : 0);
      t[2 * nb + d] = cap[d];
      t[3 * nb + d] = dev_n(d);
    }
    return launch_fetch_pools(m_table + (size_t)at * 4 * nb, table, nb, st);
  };
  // Waits for the scan's words of superstep `seq`: the totals and minimum hops
  // are then on the host, usually while the scatter still runs.
  auto wait_totals = [&](uint16_t seq) -> cudaError_t {
    uint32_t d = 0;
    for (uint32_t spin = 1, idle = 0; d < nb; ++spin) {
      const uint64_t w = h_moved[d];
      if ((uint16_t)(w >> 48) == seq) {
        h_totals[d] = (uint32_t)w;
        h_minhop[d] = (uint32_t)(w >> 32) & 0xffffu;
        ++d;
        continue;
      }
      if (spin & 0xfff) continue;
      const cudaError_t q = cudaStreamQuery(st);  // a failed or finished stream ends the wait
      if (q == cudaErrorNotReady) cudaGetLastError();  // not an error of a later launch
      else if (q != cudaSuccess) return q;
      else if (++idle > 2) return cudaErrorUnknown;
    }
    return cudaSuccess;
  };
  cudaEventRecord(t0, st);
  uint64_t superstep = 0;
  cudaError_t e = cudaSuccess;
  // The scatter of superstep k is left queued: the host next waits on the
  // stream for the partition totals of superstep k + 1, which orders it.
  bool pending = false;
  bool stale = true;  // the device's pool table is behind the host's
  while (walksum > 0 && e == cudaSuccess &&
         (p->max_supersteps == 0 || superstep < p->max_supersteps)) {
    uint32_t b;
    if (restricted) {  // the policy sees the owned blocks only
      own_num.assign(nb, 0);
      own_min.assign(nb, 0xffff);
      for (uint32_t q = own_lo; q < own_hi; ++q) {
        own_num[q] = ctx->pool_size[q];
        own_min[q] = ctx->minstep[q];
      }
      b = choose_block(own_num, own_min, p->prob, p->seed, superstep);
    } else {
      b = choose_block(ctx->pool_size, ctx->minstep, p->prob, p->seed, superstep);
    }
    const uint64_t n = ctx->pool_size[b];
    if (n == 0) return ctx->fail(GW_E_STATE, "scheduler chose an empty block (walksum %llu)",
                                 (unsigned long long)walksum);
    if (ctx->pool_host_n[b]) {
      // readWalksfromDisk: the pool's host part (its older walks) goes first,
      // then the walks that arrived on the device since it moved out.  Its
      // chunks return to the arena at once: whatever reuses them next is a
      // copy queued on st behind these.
      const uint64_t hn = ctx->pool_host_n[b], dn = n - hn;
      const uint64_t ncap = std::max<uint64_t>(n, 1024);
      void* np = nullptr;
      e = cudaMallocAsync(&np, ncap * sizeof(gw_walk_rec), st);
      if (e != cudaSuccess) break;
      for (uint64_t i = 0; i * kChunk < hn && e == cudaSuccess; ++i) {
        const uint64_t c = ctx->pool_chunks[b][i], m = std::min(kChunk, hn - i * kChunk);
        e = cudaMemcpyAsync(static_cast<gw_walk_rec*>(np) + i * kChunk, arena + c * kChunk, m * sizeof(gw_walk_rec),
                            cudaMemcpyHostToDevice, st);
      }
      if (e == cudaSuccess && dn)
        e = cudaMemcpyAsync(static_cast<gw_walk_rec*>(np) + hn, ctx->pools[b].p, dn * sizeof(gw_walk_rec),
                            cudaMemcpyDeviceToDevice, st);
      retire(b, &evs.retired);
      pool_async[b] = 1;
      ctx->pools[b].p = np;
      ctx->pools[b].bytes = ncap * sizeof(gw_walk_rec);
      cap[b] = ncap;
      for (uint32_t c : ctx->pool_chunks[b]) ctx->arena_free.push_back(c);
      ctx->pool_chunks[b].clear();
      ctx->pool_host_n[b] = 0;
      ctx->stats.pools_refilled++;
      stale = true;
      if (e != cudaSuccess) break;
    }
    WalkArgs ab = a;
    ab.lo = ctx->blocks[b];
    ab.hi = ctx->blocks[b + 1];
    const unsigned long long* beg_pos = nullptr;
    const uint32_t* csr = nullptr;
    int slot = -1;
    const PartitionPlan plan = partition_plan(n, nb);
    const size_t hist_bytes = (size_t)nb * plan.ntiles * 4;
    if (pending && (n * 4 > ctx->d_dest.bytes || hist_bytes > ctx->d_tile_hist.bytes)) {
      // a buffer the queued scatter reads is about to be replaced
      e = cudaStreamSynchronize(st);
      if (e != cudaSuccess) break;
    }
    GW_CUDA(ctx, ctx->d_dest.grow(n * 4), "dest alloc");
    GW_CUDA(ctx, ctx->d_tile_hist.grow(hist_bytes), "hist alloc");
    ps.dest = ctx->d_dest.as<uint32_t>();
    ps.tile_hist = ctx->d_tile_hist.as<uint32_t>();
    if (stale) {
      e = upload_table(0, nullptr);
      if (e != cudaSuccess) break;
      stale = false;
    }
    bool waits = false;  // the walk kernel waits for its block's copy
    if (streaming) {
      ahead.erase(std::remove(ahead.begin(), ahead.end(), b), ahead.end());
      beg_pos = ctx->d_rowptr.as<unsigned long long>() + ab.lo;
      if (slot_of[b] < 0 && n <= mapped_limit(b)) {
        csr = m_colidx + ctx->h_rowptr.as<uint64_t>()[ab.lo];
        ctx->stats.mapped_supersteps++;
        ctx->stats.mapped_walks += n;
      } else {
        slot = load_block(b, -1);
        waits = cudaEventQuery(slots.ready[slot]) == cudaErrorNotReady;
        cudaGetLastError();  // "not ready" is no error of the launches below
        if (waits) cudaEventRecord(evs.e[2], st);
        cudaStreamWaitEvent(st, slots.ready[slot], 0);
        if (waits) cudaEventRecord(evs.e[3], st);
        csr = slots.csr[slot].as<uint32_t>();
      }
    }
    // ---- exec_updates ----
    e = launch_walk_block((int)p->rule, (int)p->sink, p->aggregate != 0, ctx->pools[b].as<gw_walk_rec>(),
                          n, ctx->view(), beg_pos, csr, ab, sv, ctx->d_blocks.as<uint32_t>(), plan, ps,
                          ctx->d_status.as<uint32_t>(), st);
    if (e != cudaSuccess) break;
    if (slot >= 0) cudaEventRecord(slots.free_ev[slot], st);
    // ---- moveWalk: stable partition by destination block ----
    const uint16_t seq = (uint16_t)(superstep + 1);
    e = launch_partition_scan(plan, ps, table, b, m_moved, seq, st);
    if (e == cudaSuccess)
      e = launch_partition_scatter(ctx->pools[b].as<gw_walk_rec>(), n, plan, ps, table.ptr, table.place, table.full, st);
    if (e != cudaSuccess) break;
    if (streaming) {
      // Copy ahead: keep up to kCopyAhead blocks copied before their turn,
      // so the host link stays busy while blocks in slots run.  The candidate
      // is the block in no slot with the most pending walks (more than it
      // needs to be read in place); it takes the room of the slot with the
      // fewest pending walks, and only when it has more.
      while (ahead.size() < kCopyAhead) {
        uint64_t best = 0;
        uint32_t nxt = kNoBlock;
        for (uint32_t q = 0; q < nb; ++q)
          if (q != b && slot_of[q] < 0 && ctx->pool_size[q] > best && ctx->pool_size[q] > mapped_limit(q)) {
            best = ctx->pool_size[q];
            nxt = q;
          }
        if (nxt == kNoBlock) break;
        bool room = false;
        uint64_t minw = ~0ull;
        for (uint32_t i = 0; i < nslots; ++i) {
          if ((int)i == slot) continue;
          if (slot_block[i] == kNoBlock) room = true;
          else minw = std::min<uint64_t>(minw, ctx->pool_size[slot_block[i]]);
        }
        if (!room && best <= minw) break;
        load_block(nxt, slot);
        ahead.push_back(nxt);
      }
    }
    e = wait_totals(seq);
    if (e != cudaSuccess) break;
    if (waits) {
      float ms = 0.f;
      cudaEventElapsedTime(&ms, evs.e[2], evs.e[3]);
      ms_copy_wait += ms;
    }
    // updateWalkNum: pools too small for their new walks grow, and the
    // scatter, which has found the same and done nothing, runs again
    bool grown = false;
    ctx->pool_size[b] = 0;
    for (uint32_t d = 0; d < nb; ++d) {
      const uint64_t held = dev_n(d);  // the device part; a host part stays where it is
      const uint64_t need = held + h_totals[d];
      if (need <= cap[d]) continue;
      grown = true;
      uint64_t ncap = std::max<uint64_t>({need, cap[d] * 2, 1024});
      void* np = nullptr;
      e = cudaMallocAsync(&np, ncap * sizeof(gw_walk_rec), st);
      if (e != cudaSuccess) break;
      if (held)
        e = cudaMemcpyAsync(np, ctx->pools[d].p, held * sizeof(gw_walk_rec), cudaMemcpyDeviceToDevice, st);
      retire(d, &evs.retired);
      pool_async[d] = 1;
      ctx->pools[d].p = np;
      ctx->pools[d].bytes = ncap * sizeof(gw_walk_rec);
      cap[d] = ncap;
      if (e != cudaSuccess) break;
    }
    if (e == cudaSuccess && grown) {
      e = upload_table(1, h_totals.data());
      if (e == cudaSuccess)
        e = launch_partition_scatter(ctx->pools[b].as<gw_walk_rec>(), n, plan, ps, table.ptr, table.place, table.full,
                                     st);
    }
    if (e != cudaSuccess) break;
    pending = true;
    uint64_t forwarded = 0;
    for (uint32_t d = 0; d < nb; ++d) {
      if (!h_totals[d]) continue;
      ctx->pool_size[d] += h_totals[d];
      if (d >= own_lo && d < own_hi) forwarded += h_totals[d];
      ctx->minstep[d] = std::min<uint32_t>(ctx->minstep[d], h_minhop[d]);
    }
    walksum = walksum - n + forwarded;
    ctx->minstep[b] = 0xffff;
    ++superstep;
    e = spill_to_budget(&stale);
  }
  cudaEventRecord(t1, st);
  if (e != cudaSuccess) return ctx->cuda_fail(e, "blocked engine");
  struct {
    uint32_t full, unused;
    unsigned long long clock[kClockWords];
  } last = {};  // the end of the pool table's buffer
  GW_CUDA(ctx, cudaMemcpyAsync(&last, table.full, sizeof last, cudaMemcpyDeviceToHost, st), "clock read");
  s = take_status(ctx, st);  // synchronises the stream
  if (s == GW_OK && last.full) s = ctx->fail(GW_E_STATE, "a superstep's walks were left unplaced");
  float ms = 0.f;
  cudaEventElapsedTime(&ms, t0, t1);
  ctx->stats.supersteps = superstep;
  ctx->stats.ms_total = ms;
  // the device's clock: from the walk kernel's first CTA to the scan's, and from there to the scatter's last
  if (last.clock[kScatterEnd] > last.clock[kPartStart])
    last.clock[kPartSum] += last.clock[kScatterEnd] - last.clock[kPartStart];
  ctx->stats.ms_walk = last.clock[kWalkSum] * 1e-6;
  ctx->stats.ms_partition = last.clock[kPartSum] * 1e-6;
  ctx->stats.ms_copy_wait = ms_copy_wait;
  ctx->last_nwalks = nwalks;
  ctx->last_sink = p->sink;
  ctx->last_stride = 0;
  ctx->have_run = true;
  return s;
}

}  // namespace gw
