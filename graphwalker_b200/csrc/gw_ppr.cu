// gw_ppr.cu -- multi-source personalized PageRank (the msppr app,
// apps/msppr.cpp:25-145): per-query visit counts and top-k lists.
//
// Query q has a source vertex and a budget of walks.  Walk j of the whole
// batch belongs to the query whose prefix range holds j, starts at that
// query's source with hop 0 and uses j as its Philox stream id, so a query's
// walks are the same whether it runs alone or inside any batch.
//
// Visits go to a per-query open-addressing table of 64-bit slots
// ((tag | vertex) << 32 | count; all-ones = empty) -- the sparse replacement
// of msppr's per-source DiscreteDistribution (discretedistribution.hpp:44-57).
// The tag, in the vertex word's bits above the largest vertex id, names the
// batch that wrote the slot: a batch treats the slots of earlier batches as
// free, so its tables need no clearing pass.
// Lanes of a warp that visit the same (query, vertex) in the same step are
// folded into one table update, and the hop-0 visits of a query's walks (all
// at its source) are added in one update.  Warps take walks in small chunks
// of consecutive batch positions from a global cursor, so the walks in flight
// belong to a narrow window of queries whose tables stay in L2.
//
// Top-k: a CTA ranks a table (or a segment of one) by keys count << 32 |
// ~vertex.  Up to a few thousand slots it holds them in registers and selects
// by radix; more stream through a candidate buffer: whenever the buffer could
// overflow it is cut to the best k, and the k-th key becomes the admission
// threshold.  Large tables are split into segments ranked by separate CTAs,
// whose lists a second kernel (or, for a few queries, each query's last CTA)
// merges.  The result is the exact top k by count, ties broken by the smaller
// vertex id.
#include "gw_ppr.h"

namespace gw {

namespace {

constexpr unsigned long long kEmptySlot = ~0ull;

// Longest probe sequence an update walks before it reports the table full:
// bounds the cost of a filling table (whose query is then rerun with a larger
// one) instead of letting every further update scan the whole table.
constexpr uint32_t kMaxProbes = 256;

__device__ __forceinline__ uint32_t probe_limit(uint32_t mask) { return mask < kMaxProbes ? mask : kMaxProbes - 1; }

__device__ __forceinline__ uint32_t slot_hash(uint32_t v) {  // MurmurHash3 fmix32 (Appleby)
  v ^= v >> 16;
  v *= 0x85ebca6bu;
  v ^= v >> 13;
  v *= 0xc2b2ae35u;
  v ^= v >> 16;
  return v;
}

// Slot operations.  The load and the add carry an L2 eviction policy: the
// tables of the queries in flight should stay in L2 while the graph streams
// through it (the compare-and-swap form of atom takes none).
__device__ __forceinline__ unsigned long long load_slot(const unsigned long long* a, uint64_t pol) {
  unsigned long long r;
  asm volatile("ld.relaxed.gpu.global.L2::cache_hint.b64 %0, [%1], %2;" : "=l"(r) : "l"(a), "l"(pol) : "memory");
  return r;
}

__device__ __forceinline__ unsigned long long cas_u64(unsigned long long* a, unsigned long long cmp,
                                                      unsigned long long val) {
  unsigned long long old;
  asm volatile("atom.relaxed.gpu.global.cas.b64 %0, [%1], %2, %3;" : "=l"(old) : "l"(a), "l"(cmp), "l"(val)
               : "memory");
  return old;
}

__device__ __forceinline__ void red_add_u64(unsigned long long* a, unsigned long long v, uint64_t pol) {
  asm volatile("red.relaxed.gpu.global.add.L2::cache_hint.u64 [%0], %1, %2;" ::"l"(a), "l"(v), "l"(pol)
               : "memory");
}

// A slot another batch wrote (or never written): free for this one.
__device__ __forceinline__ bool slot_free(unsigned long long old, uint32_t tag, uint32_t tag_mask) {
  return old == kEmptySlot || ((uint32_t)(old >> 32) & tag_mask) != tag;
}

// Where v's probes in query q's table start.
__device__ __forceinline__ unsigned long long* first_slot(const QueryView& qv, uint32_t q, uint32_t v) {
  return qv.tables + __ldg(qv.table_off + q) + (slot_hash(v) & __ldg(qv.table_mask + q));
}

// R table updates per lane, side by side: update r adds n[r] visits (0: none)
// under tag | v[r] to query q[r]'s table, whose first slot was loaded as
// seen[r].  Every round acts on each update's slot as it was last seen: an add
// if it holds the key (keys stay once written), a CAS of the seen content if it
// is free or left by an earlier batch, else the next slot is loaded (linear
// probing); the rounds of the R updates overlap.  Loading a slot first costs an
// atomic only where the slot changes: a CAS of the empty pattern as the first
// probe failed on every known key and every earlier batch's slot, so nearly
// every visit took two atomics.  A table without a free slot or the key within
// kMaxProbes is reported full.
template <int R>
__device__ __forceinline__ void table_updates(const QueryView& qv, const uint32_t (&q)[R], const uint32_t (&v)[R],
                                              uint32_t (&n)[R], unsigned long long (&seen)[R], uint64_t pol) {
  unsigned long long* at[R];
#pragma unroll
  for (int r = 0; r < R; ++r) at[r] = n[r] ? first_slot(qv, q[r], v[r]) : nullptr;
  for (;;) {
    unsigned long long got[R];
    bool tried[R];  // a CAS was issued
#pragma unroll
    for (int r = 0; r < R; ++r) {
      tried[r] = false;
      got[r] = 0;
      if (n[r]) {
        const uint32_t key = qv.tag | v[r];
        if ((uint32_t)(seen[r] >> 32) == key) {
          red_add_u64(at[r], n[r], pol);
          n[r] = 0;
        } else if (slot_free(seen[r], qv.tag, qv.tag_mask)) {
          tried[r] = true;
          got[r] = cas_u64(at[r], seen[r], ((unsigned long long)key << 32) | n[r]);
        } else {
          unsigned long long* const t = qv.tables + __ldg(qv.table_off + q[r]);
          const uint32_t mask = __ldg(qv.table_mask + q[r]), slot = (uint32_t)(at[r] - t);
          if (((slot - slot_hash(v[r])) & mask) >= probe_limit(mask)) {
            qv.full[q[r]] = 1u;
            n[r] = 0;
          } else {
            at[r] = t + ((slot + 1) & mask);
            got[r] = load_slot(at[r], pol);
          }
        }
      }
    }
    uint32_t left = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (tried[r] && got[r] == seen[r]) n[r] = 0;
      seen[r] = got[r];  // another lane's claim, or the next slot
      left |= n[r];
    }
    if (!left) break;
  }
}

__device__ __forceinline__ uint32_t query_of(const unsigned long long* __restrict__ prefix, uint32_t nq,
                                             unsigned long long j) {
  uint32_t lo = 0, hi = nq - 1;  // last q with prefix[q] <= j
  while (lo < hi) {
    const uint32_t mid = (lo + hi + 1) >> 1;
    if (__ldg(prefix + mid) <= j) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

constexpr int kSmall = 0, kMid = 1, kLarge = 2;

// One walk per lane.  A visit's table update is a chain of its own (the slot,
// then a CAS or more probes), and in a warp of 32 visits some lane always has a
// long one, so the hop does not wait for it:
//
//  * kMid and kLarge, launches that fill the GPU, which the random line fills and
//    the tables' requests bound: the slot is loaded at a visit and acted on at
//    the lane's next one, behind that visit's gather.
//  * kSmall, launches of few walks, which the chain of hops bounds: visits
//    go to a queue in shared memory, worked off kFlush at a time, kPerLane per
//    lane side by side, behind a gather; the draws of the next hop are computed
//    while this one's gather is in flight, so a hop's own chain is the gather,
//    a modulo and the next address.  (It holds visits back, so the tables of
//    more queries are open at once: 16.5 ms where the others take 11.7 and 10.9 on 4096
//    queries.)
//
// Measured on B200 (walk kernel alone): 4096 queries, 59 M walks, R-MAT scale
// 24: 14.0 ms when a CAS was the first probe and the hop waited for it, 10.9
// now (35 G visits/s); one query of 100,000 walks at scale 20: 65 -> 60 us; one
// of 300 walks at scale 22: 55 -> 33 us (42 with kMid).
template <int RULE, bool ER, int SHAPE>
__global__ void __launch_bounds__(kPprThreads, SHAPE == kSmall ? 4 : SHAPE == kLarge ? 5 : 1)
    walk_query_kernel(QueryView qv, unsigned long long w_begin, unsigned long long w_end, GraphView g,
                      WalkArgs a, uint32_t* __restrict__ status) {
  constexpr bool SMALL = SHAPE == kSmall;
  constexpr int kPerLane = 2;
  constexpr uint32_t kFlush = 32 * kPerLane;
  let_next_start();
  wait_for_previous();
  __shared__ uint2 queues[SMALL ? kPprThreads / 32 : 1][kFlush + 32];  // (query, vertex)
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t below = (1u << lane) - 1u;  // lanes under this one
  uint2* const queue = queues[SMALL ? threadIdx.x >> 5 : 0];
  uint32_t queued = 0;  // warp-uniform
  const unsigned long long total = w_end - w_begin;
  const unsigned long long chunk = qv.chunk ? qv.chunk : kWarpChunk;
  const L2Hints hp = make_hints(a.hints);
  // Every walk visits its source at hop 0: the first walk of each query in
  // this launch adds all of them at once and the walks skip that update.
  const bool visits_source =
      !(rule_capped<RULE>() && a.L == 0) && !(RULE == GW_RULE_PROB && a.max_hops == 0);
  unsigned long long c_next = 0, c_end = 0;  // the warp's current chunk of batch positions
  bool drained = false;                      // the cursor has run past the batch (warp-uniform)
  bool busy = false;                         // this lane holds a walk
  unsigned long long j = 0, id_shift = 0, q_lo = 1, q_hi = 0;
  unsigned long long cur_rec = 0, src_rec = 0;  // edge-record mode: records of v and of the source
  uint32_t q = 0, src = 0, sid = 0, v = 0, hop = 0, st = 0, nvisit = 0;
  Draws dr{0, 0};
  DrawCache dc;
  dc.reset();
  // The queue's last `count` entries; equal (query, vertex) of a row of 32
  // fold into one update.
  auto flush = [&](uint32_t count) {
    __syncwarp();
    uint32_t fq[kPerLane], fv[kPerLane], fn[kPerLane];
    unsigned long long seen[kPerLane];
#pragma unroll
    for (int r = 0; r < kPerLane; ++r) {
      const uint32_t x = r * 32 + lane;
      const bool in = x < count;
      const uint2 e = in ? queue[queued - count + x] : make_uint2(0xffffffffu, lane);
      fq[r] = e.x;
      fv[r] = e.y;
      const uint32_t peers = __match_any_sync(~0u, ((unsigned long long)e.x << 32) | e.y);
      fn[r] = in && (peers & below) == 0 ? (uint32_t)__popc(peers) : 0u;
      seen[r] = fn[r] ? load_slot(first_slot(qv, fq[r], fv[r]), hp.cnt) : 0ull;
    }
    queued -= count;
    table_updates<kPerLane>(qv, fq, fv, fn, seen, hp.cnt);
    __syncwarp();
  };
  // The lane's update in flight (not SMALL).
  uint32_t p_q[1] = {0}, p_v[1] = {0}, p_n[1] = {0};
  unsigned long long p_seen[1] = {0};
  for (;;) {
    // Idle lanes take the next walks of the warp's chunk, in lane order.
    uint32_t idle = __ballot_sync(~0u, !busy);
    while (idle && !drained) {
      if (c_next >= c_end) {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(qv.cursor, chunk);
        base = __shfl_sync(~0u, base, 0);
        if (base >= total) {
          drained = true;
          break;
        }
        c_next = base;
        c_end = base + chunk < total ? base + chunk : total;
      }
      const unsigned long long avail = c_end - c_next;
      if (!busy && __popc(idle & below) < avail) {
        j = w_begin + c_next + __popc(idle & below);
        busy = true;
        if (j < q_lo || j >= q_hi) {
          q = query_of(qv.walk_prefix, qv.nq, j);
          q_lo = __ldg(qv.walk_prefix + q);
          q_hi = __ldg(qv.walk_prefix + q + 1);
          src = __ldg(qv.sources + q);
          // stream id = the walk's position in the original batch
          id_shift = qv.id_base ? __ldg(qv.id_base + q) - q_lo : 0ull;
          sid = qv.stream ? __ldg(qv.stream + q) : 0u;
          if (ER) src_rec = vertex_rec(g, hp, src);
        }
        const unsigned long long lo = q_lo > w_begin ? q_lo : w_begin, hi = q_hi < w_end ? q_hi : w_end;
        if (visits_source && j == lo && src < g.nv) {
          const uint32_t uq[1] = {q}, uv[1] = {src};
          uint32_t un[1] = {(uint32_t)(hi - lo)};
          unsigned long long seen[1] = {load_slot(first_slot(qv, q, src), hp.cnt)};
          table_updates<1>(qv, uq, uv, un, seen, hp.cnt);
        }
        v = src;
        cur_rec = src_rec;
        hop = 0;
        dc.reset();
        if (SMALL) dr = hop_draws(a, (uint32_t)(j + id_shift), 0u, sid, dc);
      }
      const uint32_t n_idle = __popc(idle);
      c_next += n_idle < avail ? n_idle : avail;
      idle = __ballot_sync(~0u, !busy);
    }
    if (!__any_sync(~0u, busy)) break;
    bool visits = false, end = true;
    if (busy) {
      if (rule_capped<RULE>() && hop >= a.L) {
      } else if (RULE == GW_RULE_PROB && hop >= a.max_hops) {
        st |= kStHops;
      } else if (v >= g.nv) {
        st |= kStBounds;
      } else {
        visits = true;
      }
    }
    const uint32_t pushes = SMALL ? __ballot_sync(~0u, visits && hop > 0) : 0u;
    if (visits) {
      ++nvisit;
      uint32_t u_n = 0;  // not SMALL: this visit's update, if the lane makes it
      const uint32_t u_v = v;
      unsigned long long u_seen = 0;
      if (SMALL) {
        if (hop > 0) queue[queued + __popc(pushes & below)] = make_uint2(q, v);
      } else if (hop > 0) {
        // lanes visiting the same (query, vertex) fold into one
        const uint32_t peers = __match_any_sync(__activemask(), ((unsigned long long)q << 32) | v);
        if ((peers & below) == 0) {
          u_n = (uint32_t)__popc(peers);
          u_seen = load_slot(first_slot(qv, q, v), hp.cnt);
        }
      }
      // the move after a walk's last visit is never observed: skipped
      if (!last_visit<RULE>(a, hop)) {
        // hop_advance_rec's choices on this hop's draws
        const unsigned long long rec = ER ? cur_rec : ld_nc_u64(g.vrec + v, hp.rec);
        if (!SMALL) dr = hop_draws(a, (uint32_t)(j + id_shift), hop, sid, dc);
        const uint32_t d0 = dr.d0, d1 = dr.d1;
        bool moved = true;
        unsigned long long off = rec >> kDegBits, deg = rec & kDegEscape;
        if (deg == kDegEscape) {
          off = __ldg(g.rowptr + v);
          deg = __ldg(g.rowptr + v + 1) - off;
        }
        if (deg > 0 && d0 >= a.thr) {
          const unsigned long long r =
              deg > 0x7fffffffull ? (unsigned long long)d1 : (unsigned long long)(d1 % (uint32_t)deg);
          if (ER) {
            const ulonglong2 e = ld_nc_u64x2(g.erec + off + r, hp.col);
            v = (uint32_t)e.y;
            cur_rec = e.x;
          } else {
            v = ld_nc_u32(g.colidx + off + r, hp.col);
          }
        } else {
          const uint32_t dj = deg > 0 ? d1 : d0;
          if (RULE == GW_RULE_JUMP) {
            v = dj % a.njump;
            if (ER) cur_rec = jump_rec(g, hp, v);
          } else if (RULE == GW_RULE_RESTART || (RULE == GW_RULE_PPR && deg == 0)) {
            v = src;
            cur_rec = src_rec;
          } else {
            moved = false;
          }
        }
        if (moved) {
          ++hop;
          end = RULE == GW_RULE_RESTART && hop % a.L == a.L - 1;
          if (SMALL && !end && !last_visit<RULE>(a, hop)) dr = hop_draws(a, (uint32_t)(j + id_shift), hop, sid, dc);
        }
      }
      if (!SMALL) {
        if (p_n[0]) table_updates<1>(qv, p_q, p_v, p_n, p_seen, hp.cnt);
        p_q[0] = q;
        p_v[0] = u_v;
        p_n[0] = u_n;
        p_seen[0] = u_seen;
      }
    }
    if (end) busy = false;
    if (SMALL) {
      queued += __popc(pushes);
      if (queued >= kFlush) flush(kFlush);
    }
  }
  if (SMALL && queued) flush(queued);
  if (!SMALL && p_n[0]) table_updates<1>(qv, p_q, p_v, p_n, p_seen, hp.cnt);
  if (st) atomicOr(status, st);
  if (qv.visits) {
    const unsigned long long w = __reduce_add_sync(~0u, nvisit);
    if (lane == 0 && w) atomicAdd(qv.visits, w);
  }
}

// Cuts cand[0, nc) (distinct nonzero keys, nc > k) to its k largest, in any
// order, at cand[0, *kept), and returns the smallest of them.  The k-th
// largest key is found by an MSB-first radix select on 8-bit digits (a
// histogram of the keys that match the digits chosen so far, one warp picks
// the digit holding rank k), which stops early once the wanted key is the
// smallest of its bucket; one compaction pass then keeps the keys >= it.
// Costs about 3 barriers per digit, where a bitonic sort of the buffer
// takes 55.
__device__ unsigned long long cut_to_k(unsigned long long* cand, uint32_t nc, uint32_t k, uint32_t* kept_out) {
  __shared__ uint32_t hist[256];
  __shared__ uint32_t sel[3];  // chosen digit, rank left inside it, keys in its bucket
  __shared__ unsigned long long kth;
  __shared__ uint32_t kept;
  const uint32_t lane = threadIdx.x & 31;
  unsigned long long prefix = 0, pmask = 0;
  uint32_t need = k;  // rank (1 = largest) of the wanted key among those matching prefix
  bool smallest_of_bucket = false;
  for (int shift = 56; shift >= 0 && !smallest_of_bucket; shift -= 8) {
    for (uint32_t b = threadIdx.x; b < 256; b += blockDim.x) hist[b] = 0;
    __syncthreads();
    for (uint32_t x = threadIdx.x; x < nc; x += blockDim.x) {
      const unsigned long long key = cand[x];
      if ((key & pmask) == prefix) atomicAdd(&hist[(uint32_t)(key >> shift) & 255u], 1u);
    }
    __syncthreads();
    if (threadIdx.x < 32) {  // lane l holds bins 255 - 8l down to 248 - 8l
      uint32_t sum = 0;
      for (uint32_t i = 0; i < 8; ++i) sum += hist[255 - 8 * lane - i];
      uint32_t incl = sum;  // keys in the bins of lanes 0..l
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(~0u, incl, o);
        if (lane >= (uint32_t)o) incl += y;
      }
      const uint32_t above = incl - sum;
      if (above < need && need <= incl) {
        uint32_t c = above;
        for (uint32_t i = 0; i < 8; ++i) {
          const uint32_t h = hist[255 - 8 * lane - i];
          if (c + h >= need) {
            sel[0] = 255 - 8 * lane - i;
            sel[1] = need - c;
            sel[2] = h;
            break;
          }
          c += h;
        }
      }
    }
    __syncthreads();
    prefix |= (unsigned long long)sel[0] << shift;
    pmask |= 255ull << shift;
    need = sel[1];
    smallest_of_bucket = sel[2] == need;
    __syncthreads();  // sel and hist are rewritten by the next digit
  }
  if (threadIdx.x == 0) {
    kth = smallest_of_bucket ? ~0ull : prefix;
    kept = 0;
  }
  __syncthreads();
  if (smallest_of_bucket) {
    for (uint32_t x = threadIdx.x; x < nc; x += blockDim.x) {
      const unsigned long long key = cand[x];
      if ((key & pmask) == prefix) atomicMin(&kth, key);
    }
    __syncthreads();
  }
  const unsigned long long t = kth;
  unsigned long long mine[kTopkBuffer / kTopkThreads];
#pragma unroll
  for (uint32_t i = 0; i < kTopkBuffer / kTopkThreads; ++i) {
    const uint32_t x = threadIdx.x + i * blockDim.x;
    mine[i] = x < nc ? cand[x] : 0ull;
  }
  __syncthreads();
#pragma unroll
  for (uint32_t i = 0; i < kTopkBuffer / kTopkThreads; ++i)
    if (mine[i] != 0ull && mine[i] >= t) cand[atomicAdd(&kept, 1u)] = mine[i];
  __syncthreads();
  *kept_out = kept;
  return t;
}

// The best k keys of n (key i = src.key(src.fetch(i)); 0 = no key) into cand,
// in any order; returns how many there are.  kTopkUnroll values per thread are fetched
// before any is converted (the loads issue back to back, so a large table is
// read with that many loads in flight per thread), then filtered one step of
// blockDim.x keys at a time into the candidate buffer; whenever the buffer
// could overflow it is cut to the best k (cut_to_k), and the k-th key
// becomes the admission threshold.
template <typename Src>
__device__ uint32_t block_best(Src src, uint32_t n, uint32_t k, unsigned long long* cand, uint32_t& ncand,
                           unsigned long long& thresh) {
  if (threadIdx.x == 0) {
    ncand = 0;
    thresh = 0;
  }
  __syncthreads();
  // nc: the candidate count, kept in a register by every thread alike.  The
  // shared ncand only hands out positions: a thread that already appends in
  // the next step changes it while slower threads would still be reading it
  // for the cut decision, so that decision must not read it.
  uint32_t nc = 0;
  for (uint32_t base = 0; base < n; base += blockDim.x * kTopkUnroll) {
    unsigned long long raw[kTopkUnroll];
#pragma unroll
    for (uint32_t u = 0; u < kTopkUnroll; ++u) {
      const uint32_t i = base + u * blockDim.x + threadIdx.x;
      raw[u] = i < n ? src.fetch(i) : Src::kNone;
    }
#pragma unroll
    for (uint32_t u = 0; u < kTopkUnroll; ++u) {
      const unsigned long long key = src.key(raw[u]);
      const bool take = key > thresh;
      if (take) cand[atomicAdd(&ncand, 1u)] = key;  // room for one full step is kept free below
      nc += (uint32_t)__syncthreads_count(take);
      if (nc > kTopkBuffer - blockDim.x) {  // cut to the best k before the next step
        uint32_t kept = 0;
        const unsigned long long t = cut_to_k(cand, nc, k, &kept);
        if (threadIdx.x == 0) {
          ncand = kept;
          thresh = t;
        }
        nc = kept;
        __syncthreads();
      }
    }
  }
  if (nc > k) {
    uint32_t kept = 0;
    cut_to_k(cand, nc, k, &kept);
    nc = kept;
  }
  return nc;
}

// The best k keys of n <= U * THREADS into cand (at least k entries), in any
// order; returns how many there are.  Every thread holds U keys in registers
// and the k-th largest is found by an MSB-first radix select over them, on
// 11-bit digits of the bits in which the keys differ (equal bits, such as the
// high bits of the counts and of the complemented vertex ids, cost no pass),
// which stops when the wanted keys fill their bucket.  Three barriers per
// digit, whatever n is, where block_best pays one for every blockDim.x keys
// and three per 8-bit digit of each cut.
struct SelectSmem {
  uint32_t hist[2][kSelectBins];  // one digit's counts, and the next one's, cleared meanwhile
  unsigned long long differ_or, differ_and;
  uint32_t warp_sum[32];
  uint32_t sel[3];  // chosen digit, rank left inside it, keys in its bucket
  uint32_t kept;
};

// Inclusive scan over the lanes of a warp.
__device__ __forceinline__ uint32_t warp_scan(uint32_t x, uint32_t lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(~0u, x, o);
    if (lane >= (uint32_t)o) x += y;
  }
  return x;
}

template <int THREADS, int U, typename Src>
__device__ uint32_t block_select(Src src, uint32_t n, uint32_t k, unsigned long long* cand, SelectSmem& sm) {
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long key[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const uint32_t i = u * THREADS + threadIdx.x;
    key[u] = i < n ? src.fetch(i) : Src::kNone;
  }
  if (threadIdx.x == 0) {
    sm.differ_or = 0;
    sm.differ_and = ~0ull;
    sm.kept = 0;
  }
  for (uint32_t b = threadIdx.x; b < kSelectBins; b += THREADS) sm.hist[0][b] = 0;
  unsigned long long any = 0, all = ~0ull;
  uint32_t mine = 0;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (u * THREADS >= n) break;
    key[u] = src.key(key[u]);
    if (key[u]) {
      any |= key[u];
      all &= key[u];
      ++mine;
    }
  }
  any = (unsigned long long)__reduce_or_sync(~0u, (uint32_t)(any >> 32)) << 32 | __reduce_or_sync(~0u, (uint32_t)any);
  all = (unsigned long long)__reduce_and_sync(~0u, (uint32_t)(all >> 32)) << 32 | __reduce_and_sync(~0u, (uint32_t)all);
  mine = __reduce_add_sync(~0u, mine);
  __syncthreads();
  if (lane == 0) {
    sm.warp_sum[warp] = mine;
    if (mine) {
      atomicOr(&sm.differ_or, any);
      atomicAnd(&sm.differ_and, all);
    }
  }
  __syncthreads();
  const uint32_t m = __reduce_add_sync(~0u, lane < THREADS / 32 ? sm.warp_sum[lane] : 0u);
  unsigned long long prefix = 0, pmask = 0;  // keys >= prefix are kept (all, when m <= k)
  if (m > k) {
    const unsigned long long ones = sm.differ_or, differ = ones ^ sm.differ_and;
    unsigned long long left = differ;  // differing bits not looked at yet
    uint32_t need = k;                 // rank (1 = largest) of the wanted key among those matching prefix
    bool whole = false;
    for (uint32_t t = 0; left && !whole; t ^= 1) {
      const int top = 64 - __clzll((long long)left);
      const int shift = top < kSelectBits ? 0 : top - kSelectBits;
      const uint32_t dmask = (1u << (top - shift)) - 1u;
      // the equal bits above the digit belong to the prefix
      const unsigned long long above = top < 64 ? ~0ull << top : 0ull;
      prefix |= ones & above & ~pmask;
      pmask |= above;
      uint32_t* const hist = sm.hist[t];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (u * THREADS >= n) break;
        const bool in = key[u] && (key[u] & pmask) == prefix;
        const uint32_t digit = (uint32_t)(key[u] >> shift) & dmask;
        const uint32_t zeros = __ballot_sync(~0u, in && digit == 0);  // the common digit: one update per warp
        if (lane == 0 && zeros) atomicAdd(&hist[0], (uint32_t)__popc(zeros));
        if (in && digit) atomicAdd(&hist[digit], 1u);
      }
      __syncthreads();
      // thread x holds the bins from the top: kSelectBins - 1 - kPer * x down
      constexpr uint32_t kPer = kSelectBins / THREADS;
      const uint32_t first = kSelectBins - 1 - kPer * threadIdx.x;
      uint32_t sum = 0;
#pragma unroll
      for (uint32_t i = 0; i < kPer; ++i) {
        sum += hist[first - i];
        sm.hist[t ^ 1][first - i] = 0;
      }
      const uint32_t incl = warp_scan(sum, lane);
      if (lane == 31) sm.warp_sum[warp] = incl;
      __syncthreads();
      const uint32_t warps = warp_scan(lane < THREADS / 32 ? sm.warp_sum[lane] : 0u, lane);
      const uint32_t below = __shfl_sync(~0u, warps, warp ? warp - 1 : 0);
      const uint32_t upto = incl + (warp ? below : 0u);
      uint32_t c = upto - sum;
      if (c < need && need <= upto) {
        for (uint32_t i = 0; i < kPer; ++i) {
          const uint32_t h = hist[first - i];
          if (c + h >= need) {
            sm.sel[0] = first - i;
            sm.sel[1] = need - c;
            sm.sel[2] = h;
            break;
          }
          c += h;
        }
      }
      __syncthreads();
      prefix |= (unsigned long long)sm.sel[0] << shift;
      pmask |= (unsigned long long)dmask << shift;
      need = sm.sel[1];
      whole = sm.sel[2] == need;  // the bucket's keys are all wanted
      left &= (1ull << shift) - 1ull;
    }
    // every bit below was equal or is all wanted: the prefix is the bound
    if (!whole) prefix |= ones & ~pmask;
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (u * THREADS >= n) break;
    if (key[u] && key[u] >= prefix) cand[atomicAdd(&sm.kept, 1u)] = key[u];
  }
  __syncthreads();
  return sm.kept;
}

// Key of a table slot: count << 32 | ~vertex (larger = more visits, then the
// smaller vertex id); 0 for a free slot (empty, or another batch's).  For
// kernels that start when the walks have ended: the read-only path streams
// faster than coherent loads (64 queries of 100,000 walks, k = 100: 273 us of
// top-k, 286).
struct SlotKey {
  static constexpr unsigned long long kNone = kEmptySlot;
  const unsigned long long* t;
  uint64_t pol;
  uint32_t tag, tag_mask;
  __device__ unsigned long long fetch(uint32_t i) const { return ld_nc_u64(t + i, pol); }
  __device__ unsigned long long key(unsigned long long e) const {
    return slot_free(e, tag, tag_mask) ? 0ull
                                       : ((e & 0xffffffffull) << 32) | (uint32_t)~((uint32_t)(e >> 32) & ~tag_mask);
  }
};

// The same in a kernel that was launched while the walks ran.
struct LiveSlotKey : SlotKey {
  __device__ unsigned long long fetch(uint32_t i) const { return load_slot(t + i, pol); }
};

struct CandKey {  // candidate lists hold keys already (0 = none)
  static constexpr unsigned long long kNone = 0ull;
  const unsigned long long* c;
  __device__ unsigned long long fetch(uint32_t i) const { return c[i]; }
  __device__ static unsigned long long key(unsigned long long v) { return v; }
};

// Lists that other CTAs of the same launch wrote.  (A merge in a launch of its
// own reads plainly: one query of 300,000 walks, k = 500, 593 us of top-k, 656
// with __ldcg.)
struct LiveCandKey : CandKey {
  __device__ unsigned long long fetch(uint32_t i) const { return __ldcg(c + i); }
};

// Row q of the result: the n <= k distinct keys of cand by rank, largest
// first, a key per thread counting the larger ones; then empty entries.
__device__ void write_topk(const unsigned long long* cand, uint32_t n, uint32_t q, uint32_t k, uint32_t* out_ids,
                           uint32_t* out_counts) {
  out_ids += (unsigned long long)q * k;
  out_counts += (unsigned long long)q * k;
  for (uint32_t r = threadIdx.x; r < k; r += blockDim.x) {
    const unsigned long long key = r < n ? cand[r] : 0ull;
    uint32_t rank = r;
    if (r < n) {
      rank = 0;
      for (uint32_t j = 0; j < n; ++j) rank += cand[j] > key ? 1u : 0u;
    }
    out_ids[rank] = key ? ~(uint32_t)key : 0xffffffffu;
    out_counts[rank] = (uint32_t)(key >> 32);
  }
}

// Shared memory of a ranking CTA.
struct TopkSmem {
  unsigned long long cand[kTopkBuffer];
  SelectSmem select;
  uint32_t ncand;
  unsigned long long thresh;
};

// Small tables are ranked from registers: 8 slots per thread, so that the
// streaming of the large ones keeps its three CTAs per SM.
constexpr int kSmallUnroll = 8;

__device__ uint32_t best_slots(const SlotKey& src, uint32_t n, uint32_t k, TopkSmem& sm) {
  return n <= kSmallUnroll * kTopkThreads ? block_select<kTopkThreads, kSmallUnroll>(src, n, k, sm.cand, sm.select)
                                          : block_best(src, n, k, sm.cand, sm.ncand, sm.thresh);
}

__device__ __forceinline__ SlotKey table_slots(const QueryView& qv, uint32_t q, uint32_t first) {
  return SlotKey{qv.tables + qv.table_off[q] + first, l2_policy(true, false), qv.tag, qv.tag_mask};
}

// One CTA per query over its whole table; CTA i takes query q_begin +
// order[i] (order NULL: i).
__global__ void __launch_bounds__(kTopkThreads, 3)
    topk_kernel(QueryView qv, uint32_t q_begin, uint32_t k, const uint32_t* __restrict__ order,
                uint32_t* __restrict__ out_ids, uint32_t* __restrict__ out_counts) {
  __shared__ TopkSmem sm;
  const uint32_t q = q_begin + (order ? __ldg(order + blockIdx.x) : blockIdx.x);
  const uint32_t n = best_slots(table_slots(qv, q, 0), qv.table_mask[q] + 1, k, sm);
  write_topk(sm.cand, n, q, k, out_ids, out_counts);
}

// The query holding segment g.
__device__ __forceinline__ uint32_t segment_query(const unsigned long long* __restrict__ seg_first, uint32_t lo,
                                                  uint32_t hi, unsigned long long g) {
  while (lo < hi) {
    const uint32_t mid = (lo + hi + 1) >> 1;
    if (seg_first[mid] <= g) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// One CTA per table segment of seg_slots slots (CTA i takes segment
// seg_first[q_begin] + order[i]; order NULL: i): a query with one segment
// gets its list here; the others leave their segments' best k keys in
// seg_cand for topk_merge_kernel.
__global__ void __launch_bounds__(kTopkThreads, 3)
    topk_segment_kernel(QueryView qv, uint32_t q_begin, uint32_t q_count, uint32_t k, uint32_t seg_slots,
                        const unsigned long long* __restrict__ seg_first, const uint32_t* __restrict__ order,
                        unsigned long long* __restrict__ seg_cand, uint32_t* __restrict__ out_ids,
                        uint32_t* __restrict__ out_counts) {
  __shared__ TopkSmem sm;
  const unsigned long long g = seg_first[q_begin] + (order ? __ldg(order + blockIdx.x) : blockIdx.x);
  const uint32_t q = segment_query(seg_first, q_begin, q_begin + q_count - 1, g);
  const unsigned long long nseg = seg_first[q + 1] - seg_first[q];
  const uint32_t cap = qv.table_mask[q] + 1;
  const uint32_t first = (uint32_t)(g - seg_first[q]) * seg_slots;
  const uint32_t n = best_slots(table_slots(qv, q, first), cap - first < seg_slots ? cap - first : seg_slots, k, sm);
  if (nseg == 1) {
    write_topk(sm.cand, n, q, k, out_ids, out_counts);
  } else {
    for (uint32_t r = threadIdx.x; r < k; r += blockDim.x) seg_cand[g * k + r] = r < n ? sm.cand[r] : 0ull;
  }
}

// One CTA per query with several segments: the best k of its segments' lists.
__global__ void __launch_bounds__(kTopkThreads, 3)
    topk_merge_kernel(uint32_t q_begin, uint32_t k, const unsigned long long* __restrict__ seg_first,
                      const unsigned long long* __restrict__ seg_cand, uint32_t* __restrict__ out_ids,
                      uint32_t* __restrict__ out_counts) {
  __shared__ TopkSmem sm;
  const uint32_t q = q_begin + blockIdx.x;
  const unsigned long long s0 = seg_first[q], nseg = seg_first[q + 1] - s0;
  if (nseg < 2) return;
  const CandKey src{seg_cand + s0 * k};
  const uint32_t keys = (uint32_t)(nseg * k);
  const uint32_t n = keys <= kSmallUnroll * kTopkThreads
                         ? block_select<kTopkThreads, kSmallUnroll>(src, keys, k, sm.cand, sm.select)
                         : block_best(src, keys, k, sm.cand, sm.ncand, sm.thresh);
  write_topk(sm.cand, n, q, k, out_ids, out_counts);
}

// A few queries: segments of kTopkFewSlots slots, ranked from registers, and
// the CTA that finishes a query's last segment merges its lists (at most
// kTopkFewKeys keys), so a query costs one launch.  seg_done: per query,
// segments finished (zero; left zero).
//
// One query of 100,000 walks (a million slots) took 26 us in 64 streaming CTAs
// and 22 us in the merge's one, most of it barriers; here 26 together (ncu, cold L2).
//
// It is launched to start while the walk kernel drains: what it reads before
// wait_for_previous() was copied up before that kernel.
__global__ void __launch_bounds__(kTopkFewThreads, 1)
    topk_few_kernel(QueryView qv, uint32_t q_begin, uint32_t q_count, uint32_t k,
                    const unsigned long long* __restrict__ seg_first, unsigned long long* seg_cand,
                    uint32_t* __restrict__ seg_done, uint32_t* __restrict__ out_ids,
                    uint32_t* __restrict__ out_counts) {
  __shared__ unsigned long long cand[kTopkMaxK];
  __shared__ SelectSmem select;
  __shared__ bool last;
  const unsigned long long g = seg_first[q_begin] + blockIdx.x;
  const uint32_t q = segment_query(seg_first, q_begin, q_begin + q_count - 1, g);
  const uint32_t nseg = (uint32_t)(seg_first[q + 1] - seg_first[q]);
  const uint32_t cap = qv.table_mask[q] + 1, first = (uint32_t)(g - seg_first[q]) * kTopkFewSlots;
  wait_for_previous();
  uint32_t n = block_select<kTopkFewThreads, kTopkFewSlots / kTopkFewThreads>(
      LiveSlotKey{table_slots(qv, q, first)}, cap - first < kTopkFewSlots ? cap - first : kTopkFewSlots, k, cand, select);
  if (nseg > 1) {
    for (uint32_t r = threadIdx.x; r < k; r += blockDim.x) seg_cand[g * k + r] = r < n ? cand[r] : 0ull;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
      last = atomicAdd(seg_done + q, 1u) + 1 == nseg;
      if (last) seg_done[q] = 0;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    n = block_select<kTopkFewThreads, kTopkFewKeys / kTopkFewThreads>(LiveCandKey{{seg_cand + seg_first[q] * k}},
                                                                      nseg * k, k, cand, select);
  }
  write_topk(cand, n, q, k, out_ids, out_counts);
}

__global__ void clear_tables_kernel(ulonglong2* __restrict__ t, unsigned long long n2) {
  const ulonglong2 empty = make_ulonglong2(kEmptySlot, kEmptySlot);
  let_next_start();
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < n2;
       i += (unsigned long long)gridDim.x * blockDim.x)
    t[i] = empty;
}

// One CTA per piece of a query's table (tables are powers of two of at least
// 256 slots).
__global__ void __launch_bounds__(256)
    clear_queries_kernel(QueryView qv, const unsigned long long* __restrict__ piece_first) {
  let_next_start();
  const uint32_t q = segment_query(piece_first, 0, qv.nq - 1, blockIdx.x);
  const uint32_t slots = qv.table_mask[q] + 1, first = (uint32_t)(blockIdx.x - piece_first[q]) * kClearSlots;
  const uint32_t n2 = (slots - first < kClearSlots ? slots - first : kClearSlots) / 2;
  ulonglong2* const t = reinterpret_cast<ulonglong2*>(qv.tables + qv.table_off[q] + first);
  for (uint32_t i = threadIdx.x; i < n2; i += 256) t[i] = make_ulonglong2(kEmptySlot, kEmptySlot);
}

int sm_count() {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

// Launches up to this many walks run the kSmall kernel: one CTA per SM.  Scales
// 20 and 22, one query: 3000 walks 41 us against 49, 20,000 42.5 against 46.5,
// 37,000 45 against 48, 60,000 54 against 53, 100,000 76 against 60.
constexpr unsigned long long kSmallLaunch = 148 * kPprThreads;
// From here on the kLarge kernel: the same in 51 registers, five CTAs per SM
// instead of four (4096 queries 10.9 ms against 11.7; 4.1 M walks at scale 22
// 0.80 against 0.85; 600,000 at 23 0.19 against 0.18).
constexpr unsigned long long kLargeLaunch = 1u << 20;

template <int RULE>
cudaError_t query_dispatch(const QueryView& qv, unsigned long long w_begin, unsigned long long w_end,
                           const GraphView& g, const WalkArgs& a, uint32_t* status, int threads_per_sm,
                           cudaStream_t stream) {
  const unsigned long long n = w_end - w_begin;
  const int shape = n <= kSmallLaunch ? kSmall : n < kLargeLaunch ? kMid : kLarge;
  auto kern = g.erec ? (shape == kSmall  ? walk_query_kernel<RULE, true, kSmall>
                        : shape == kMid ? walk_query_kernel<RULE, true, kMid>
                                        : walk_query_kernel<RULE, true, kLarge>)
                     : (shape == kSmall  ? walk_query_kernel<RULE, false, kSmall>
                        : shape == kMid ? walk_query_kernel<RULE, false, kMid>
                                        : walk_query_kernel<RULE, false, kLarge>);
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kPprThreads, 0);
  const int sms = sm_count();
  if (per_sm <= 0) per_sm = 1;
  if (threads_per_sm > 0) per_sm = std::max(1, std::min(per_sm, threads_per_sm / kPprThreads));
  const unsigned long long need = (n + kPprThreads - 1) / kPprThreads;
  const unsigned long long full = (unsigned long long)sms * per_sm;
  const int grid = (int)(need < full ? (need ? need : 1) : full);
  // Walks per cursor grab: no larger than gives every warp of the grid a
  // share, so a launch of few walks (one query, a small serving step) runs
  // them side by side instead of a lane's worth of walks one after another.
  QueryView q = qv;
  const unsigned long long warps = (unsigned long long)grid * (kPprThreads / 32);
  const unsigned long long fair = ((n + warps - 1) / warps + 31) / 32 * 32;
  const unsigned long long chunk = qv.chunk ? qv.chunk : kWarpChunk;
  q.chunk = (uint32_t)(fair < chunk ? fair : chunk);
  return launch_dependent(kern, grid, kPprThreads, 0, stream, q, w_begin, w_end, g, a, status);
}

}  // namespace

cudaError_t launch_walk_queries(int rule, const QueryView& qv, unsigned long long w_begin,
                                unsigned long long w_end, const GraphView& g, const WalkArgs& a,
                                uint32_t* status, int threads_per_sm, cudaStream_t stream) {
  if (w_end <= w_begin || qv.nq == 0) return cudaSuccess;
  if (!qv.cursor) return cudaErrorInvalidValue;
  switch (rule) {
    case GW_RULE_JUMP: return query_dispatch<GW_RULE_JUMP>(qv, w_begin, w_end, g, a, status, threads_per_sm, stream);
    case GW_RULE_STOP: return query_dispatch<GW_RULE_STOP>(qv, w_begin, w_end, g, a, status, threads_per_sm, stream);
    case GW_RULE_PROB: return query_dispatch<GW_RULE_PROB>(qv, w_begin, w_end, g, a, status, threads_per_sm, stream);
    case GW_RULE_RESTART:
      return query_dispatch<GW_RULE_RESTART>(qv, w_begin, w_end, g, a, status, threads_per_sm, stream);
    case GW_RULE_PPR: return query_dispatch<GW_RULE_PPR>(qv, w_begin, w_end, g, a, status, threads_per_sm, stream);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_clear_tables(unsigned long long* tables, unsigned long long n, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  if ((reinterpret_cast<uintptr_t>(tables) & 15) || (n & 1))  // not in 16-byte pairs: byte fill
    return cudaMemsetAsync(tables, 0xff, n * sizeof(unsigned long long), stream);
  const unsigned long long n2 = n / 2, need = (n2 + 255) / 256, full = (unsigned long long)sm_count() * 32;
  clear_tables_kernel<<<(unsigned)(need < full ? need : full), 256, 0, stream>>>(
      reinterpret_cast<ulonglong2*>(tables), n2);
  return cudaGetLastError();
}

cudaError_t launch_clear_queries(const QueryView& qv, const unsigned long long* d_piece_first, uint64_t npieces,
                                 cudaStream_t stream) {
  if (npieces == 0) return cudaSuccess;
  if (npieces > 0x7fffffffull) return cudaErrorInvalidValue;
  clear_queries_kernel<<<(unsigned)npieces, 256, 0, stream>>>(qv, d_piece_first);
  return cudaGetLastError();
}

uint32_t topk_segment_slots(const uint32_t* table_mask, uint32_t nq, uint32_t k) {
  uint64_t few = 0;
  bool merged = true;  // one CTA can hold every query's lists
  for (uint32_t q = 0; q < nq && few <= kTopkFewSegments; ++q) {
    const uint64_t segments = table_mask[q] / kTopkFewSlots + 1;
    few += segments;
    merged = merged && segments * k <= kTopkFewKeys;
  }
  // Past the register path twice the segments only double what one CTA merges
  // (a call for one query of 300,000 walks, k = 500: 950 us with kTopkFewSlots,
  // 845 with kTopkSegment; k = 100: 256 and 220).
  if (few <= kTopkFewSegments && merged) return kTopkFewSlots;
  uint64_t s = kTopkSegment;
  while (s < (1ull << 30) && s / kTopkSegment * 64 < nq) s <<= 1;  // 64 queries per doubling
  return (uint32_t)s;
}

bool topk_is_few(const unsigned long long* seg_first, uint32_t nq, uint32_t seg_slots, uint32_t k) {
  // the register path pays while its CTAs (one per SM) make few waves, and one
  // CTA must be able to hold a query's lists
  if (seg_slots != kTopkFewSlots || seg_first[nq] - seg_first[0] > kTopkFewSegments) return false;
  for (uint32_t q = 0; q < nq; ++q)
    if ((seg_first[q + 1] - seg_first[q]) * k > kTopkFewKeys) return false;
  return true;
}

void topk_segment_prefix(const uint32_t* table_mask, uint32_t nq, uint32_t seg_slots, unsigned long long* seg_first) {
  seg_first[0] = 0;
  for (uint32_t q = 0; q < nq; ++q)
    seg_first[q + 1] = seg_first[q] + ((unsigned long long)table_mask[q] + seg_slots) / seg_slots;
}

void topk_segment_order(const uint32_t* table_mask, uint32_t nq, uint32_t seg_slots,
                        const unsigned long long* seg_first, uint32_t* order) {
  // a table is a power of two, so is a segment: bucket the segments by
  // log2(size), largest bucket first, each bucket in segment order
  std::vector<uint32_t> start(34, 0);
  auto bucket = [&](uint32_t q, unsigned long long i) {
    const unsigned long long cap = (unsigned long long)table_mask[q] + 1, first = i * seg_slots;
    const unsigned long long size = cap - first < seg_slots ? cap - first : seg_slots;
    return 63 - __builtin_clzll(size);  // 0..32
  };
  for (uint32_t q = 0; q < nq; ++q)
    for (unsigned long long i = 0; i < seg_first[q + 1] - seg_first[q]; ++i) ++start[32 - bucket(q, i) + 1];
  for (int b = 1; b < 34; ++b) start[b] += start[b - 1];
  for (uint32_t q = 0; q < nq; ++q)
    for (unsigned long long i = 0; i < seg_first[q + 1] - seg_first[q]; ++i)
      order[start[32 - bucket(q, i)]++] = (uint32_t)(seg_first[q] + i);
}

cudaError_t launch_topk_segmented(const QueryView& qv, uint32_t q_begin, uint32_t q_count, uint32_t k,
                                  uint32_t* out_ids, uint32_t* out_counts, const unsigned long long* d_seg_first,
                                  const unsigned long long* h_seg_first, uint32_t seg_slots,
                                  unsigned long long* d_seg_cand, uint32_t* d_seg_done, const uint32_t* d_order,
                                  cudaStream_t stream) {
  if (q_count == 0) return cudaSuccess;
  if (k == 0 || k > kTopkMaxK) return cudaErrorInvalidValue;
  const unsigned long long nseg = h_seg_first[q_begin + q_count] - h_seg_first[q_begin];
  if (nseg == 0 || nseg > 0x7fffffffull) return cudaErrorInvalidValue;
  if (topk_is_few(h_seg_first + q_begin, q_count, seg_slots, k)) {
    return launch_dependent(topk_few_kernel, (unsigned)nseg, kTopkFewThreads, 0, stream, qv, q_begin, q_count, k,
                            d_seg_first, d_seg_cand, d_seg_done, out_ids, out_counts);
  }
  if (nseg == q_count) {  // no table is split: one CTA per query
    topk_kernel<<<q_count, kTopkThreads, 0, stream>>>(qv, q_begin, k, d_order, out_ids, out_counts);
    return cudaGetLastError();
  }
  topk_segment_kernel<<<(unsigned)nseg, kTopkThreads, 0, stream>>>(qv, q_begin, q_count, k, seg_slots, d_seg_first,
                                                                    d_order, d_seg_cand, out_ids, out_counts);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess && nseg > q_count) {  // some query has several segments
    topk_merge_kernel<<<q_count, kTopkThreads, 0, stream>>>(q_begin, k, d_seg_first, d_seg_cand, out_ids, out_counts);
    e = cudaGetLastError();
  }
  return e;
}

}  // namespace gw
