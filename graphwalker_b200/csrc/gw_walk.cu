// gw_walk.cu -- the walk-advance kernels (the per-block update loop of
// GraphWalker, src/engine/graphwalker.hpp:257-270 + the updateByWalk of each
// walk class, src/walks/randomwalk*.hpp) and the 64-bit walk codec kernels
// (src/walks/walk.hpp:69-91).
//
// Resident mode: one persistent launch runs every walk to its end.  Each
// thread holds one walk and advances it one hop per loop iteration; when its
// walk ends it takes the next one (index += grid stride) inside the same
// iteration, so lanes never wait for the longest walk of their warp.  Per hop:
// one 8-byte packed vertex record load, one 4-byte column load, one Philox
// block computed while the record load is in flight, and one visit atomic.
// With edge records (ER) the record of the current vertex is carried from the
// previous hop, so a hop along an edge is a single 16-byte gather; graphs of a
// few L2 sizes are walked over the plain layout all the same
// (walks_use_records).
#include <algorithm>

#include "gw_internal.h"

namespace gw {

namespace {

__device__ __forceinline__ uint4 load_walk(const gw_walk_rec* __restrict__ walks, uint64_t i) {
  return __ldg(reinterpret_cast<const uint4*>(walks) + i);
}

// The walk record of the resident kernel, read once: with
// kHintStreamsEvictFirst it is marked to leave L2 first.
__device__ __forceinline__ uint4 load_walk_hinted(const gw_walk_rec* __restrict__ walks, uint64_t i,
                                                  const WalkArgs& a, const L2Hints& hp) {
  return (a.hints & kHintStreamsEvictFirst) ? ld_nc_u32x4(reinterpret_cast<const uint4*>(walks) + i, hp.strm)
                                            : load_walk(walks, i);
}

// A walk's start record: like vertex_rec, with the stream policy when asked.
__device__ __forceinline__ unsigned long long start_rec(const GraphView& g, const WalkArgs& a, const L2Hints& hp,
                                                        uint32_t v) {
  if (v >= g.nv) return 0ull;
  return ld_nc_u64(g.vrec + v, (a.hints & kHintStreamsEvictFirst) ? hp.strm : hp.rec);
}

template <int RULE, int SINK, bool AGG, bool ER>
__global__ void __launch_bounds__(kWalkThreads)
    walk_resident_kernel(const gw_walk_rec* __restrict__ walks, uint64_t n, GraphView g,
                         WalkArgs a, SinkView s, uint32_t* __restrict__ status) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const L2Hints hp = make_hints(a.hints);
  uint4 w = load_walk_hinted(walks, i, a, hp);
  uint32_t v = w.x, id = w.y, src = w.z, hop = w.w, k = 0;
  uint32_t st = 0;
  uint32_t clos = 0;
  DrawCache dc;
  dc.reset();
  // edge-record mode: the records of the current vertex and of the source
  unsigned long long rec = 0, src_rec = 0;
  if (ER) {
    rec = start_rec(g, a, hp, v);
    if (rule_returns<RULE>()) src_rec = src == v ? rec : vertex_rec(g, hp, src);
  }
  for (;;) {
    bool end;
    if (rule_capped<RULE>() && hop >= a.L) {
      end = true;
    } else if (RULE == GW_RULE_PROB && hop >= a.max_hops) {
      st |= kStHops;
      end = true;
    } else if (v >= g.nv) {
      st |= kStBounds;
      end = true;
    } else {
      // the app's updateInfo(src, v, tid, hop) precedes the draws
      if (SINK == GW_SINK_VERTEX_COUNT) {
        count_visit<AGG>(s.counts, v, hp.cnt);
      } else if (SINK == GW_SINK_PATH_RECORD) {
        if (k < a.path_stride) s.paths[i * a.path_stride + k] = v;
        else st |= kStOverflow;
      } else if (SINK == GW_SINK_CLOSURE_COUNT) {
        clos += ((int)hop >= (int)a.L - 1 && v == src) ? 1u : 0u;
      }
      ++k;
      if (last_visit<RULE>(a, hop)) {
        end = true;  // the move after the last visit is never observed
      } else {
        end = ER ? !hop_advance_carried<RULE>(g, a, hp, id, src, src_rec, hop, v, rec, dc)
                 : !hop_advance<RULE>(g, a, hp, id, src, hop, v, dc);
        if (!end) {
          ++hop;
          if (RULE == GW_RULE_RESTART && hop % a.L == a.L - 1) end = true;
        }
      }
    }
    if (end) {
      if (SINK == GW_SINK_PATH_RECORD) s.plen[i] = k;
      i += stride;
      if (i >= n) break;
      w = load_walk_hinted(walks, i, a, hp);
      v = w.x;
      id = w.y;
      src = w.z;
      hop = w.w;
      k = 0;
      dc.reset();
      if (ER) {
        rec = start_rec(g, a, hp, v);
        if (rule_returns<RULE>()) src_rec = src == v ? rec : vertex_rec(g, hp, src);
      }
    }
  }
  if (st) atomicOr(status, st);
  if (SINK == GW_SINK_CLOSURE_COUNT && clos) atomicAdd(s.closure, (unsigned long long)clos);
}

// Edge records: erec[e] = (packed record of colidx[e], colidx[e]).
__global__ void build_erec_kernel(const uint32_t* __restrict__ colidx, const unsigned long long* __restrict__ vrec,
                                  uint64_t ne, uint32_t nv, ulonglong2* __restrict__ erec) {
  for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < ne;
       e += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t w = __ldg(colidx + e);
    erec[e] = make_ulonglong2(w < nv ? __ldg(vrec + w) : 0ull, (unsigned long long)w);
  }
}

__device__ __forceinline__ uint32_t find_block(const uint32_t* __restrict__ blocks,
                                               uint32_t nblocks, uint32_t v) {
  // first p with v < blocks[p+1] (RandomWalk::getblock, randomwalk.hpp:74-82)
  uint32_t lo = 0, hi = nblocks;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (v < blocks[mid + 1]) hi = mid;
    else lo = mid + 1;
  }
  return lo;
}

__device__ __forceinline__ unsigned long long clock_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// Blocked-mode superstep over the walks of block [a.lo, a.hi): the in-block
// loop of updateByWalk and, on leaving, getblock + moveWalk
// (randomwalkwithjump.hpp:40-60 and siblings), with the first half of the
// stable partition by destination block folded in.
//
// One CTA owns one tile of plan.tile() consecutive walks, a row of 256 at a
// time.  After a row's walks have stopped, each walk's rank among the tile's
// earlier walks of the same destination comes from a warp match, the counts
// of the lower warps of the row and the running counts of the tile; the walk
// leaves dest = destination | rank << 16 and the tile leaves one count per
// destination, so placing the walks needs one scan of the tile counts and one
// elementwise scatter (gw_partition.cu).
//
// A superstep of a few 100,000 walks is bound by latency: the pool record, the
// vertex record and the column are three dependent loads, and every further
// launch adds its own start and tail.  A separate histogram pass over the
// walks (one warp per 256 walks, eight rows in sequence) took 10.4 us beside
// 9.6 us for the walk itself at 126 k walks and 33 blocks.
template <int RULE, int SINK, bool AGG, bool SLICE>
__global__ void __launch_bounds__(kWalkThreads)
    walk_block_kernel(gw_walk_rec* __restrict__ walks, uint64_t n, GraphView g,
                      const unsigned long long* __restrict__ beg_pos,
                      const uint32_t* __restrict__ csr, WalkArgs a, SinkView s,
                      const uint32_t* __restrict__ blocks, PartitionPlan plan, PartitionScratch ps,
                      uint32_t* __restrict__ status) {
  extern __shared__ uint32_t smem[];
  const uint32_t nb = plan.nbuckets;
  uint32_t* const total = smem;       // per destination: walks of the rows done
  uint32_t* const minhop = smem + nb; // per destination: lowest hop
  uint32_t* const sblk = smem + 2 * nb;
  const bool staged = nb <= kStagedBlocks;
  uint8_t* const wcnt = reinterpret_cast<uint8_t*>(sblk + (staged ? nb + 1 : 0));  // [warp][destination], this row
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint64_t base = (uint64_t)blockIdx.x * plan.tile();
  let_next_start();
  if (ps.clock && blockIdx.x == 0 && threadIdx.x == 0) ps.clock[kWalkStart] = clock_ns();
  uint64_t i = base + threadIdx.x;
  uint4 w = make_uint4(0, 0, 0, 0);
  if (i < n) w = *(reinterpret_cast<const uint4*>(walks) + i);
  for (uint32_t b = threadIdx.x; b < nb; b += kWalkThreads) {
    total[b] = 0;
    minhop[b] = 0xffffffffu;
  }
  for (uint32_t b = threadIdx.x; b < nb * (kWalkThreads / 32); b += kWalkThreads) wcnt[b] = 0;
  if (staged)
    for (uint32_t b = threadIdx.x; b <= nb; b += kWalkThreads) sblk[b] = __ldg(blocks + b);
  const uint32_t* const bl = staged ? sblk : blocks;
  __syncthreads();
  uint32_t st = 0, clos = 0;
  const L2Hints hp = make_hints(a.hints);
  DrawCache dc;
  // the slice's first edge index (csr[0] is edge b0); read once, since the
  // slice may be pinned host memory read over the host link
  const unsigned long long b0 = SLICE && n ? __ldg(beg_pos) : 0ull;
  for (uint32_t row = 0;;) {
    uint32_t d = kNoDest;
    uint32_t hop = 0;
    if (i < n) {
      uint32_t v = w.x;
      const uint32_t id = w.y, src = w.z;
      hop = w.w;
      bool ended = false;
      dc.reset();
      while (v >= a.lo && v < a.hi) {
        if (rule_capped<RULE>() && hop >= a.L) break;
        if (RULE == GW_RULE_PROB && hop >= a.max_hops) {
          st |= kStHops;
          ended = true;
          break;
        }
        if (v >= g.nv) {
          st |= kStBounds;
          ended = true;
          break;
        }
        if (SINK == GW_SINK_VERTEX_COUNT) count_visit<AGG>(s.counts, v, hp.cnt);
        else if (SINK == GW_SINK_CLOSURE_COUNT)
          clos += ((int)hop >= (int)a.L - 1 && v == src) ? 1u : 0u;
        if (last_visit<RULE>(a, hop)) {  // its move is never observed: the walk ends here
          ++hop;
          ended = true;
          break;
        }
        bool moved;
        if (SLICE) moved = hop_advance_slice<RULE>(beg_pos, csr, b0, a, id, src, hop, v, dc);
        else moved = hop_advance<RULE>(g, a, hp, id, src, hop, v, dc);
        if (!moved) {
          ended = true;
          break;
        }
        ++hop;
        if (RULE == GW_RULE_RESTART && hop % a.L == a.L - 1) {
          ended = true;
          break;
        }
      }
      if (!ended) {
        bool alive;
        if (rule_capped<RULE>()) alive = hop < a.L;
        else if (RULE == GW_RULE_RESTART) alive = hop % a.L != a.L - 1;
        else alive = true;
        if (alive) {
          const uint32_t to = find_block(bl, nb, v);
          if (to < nb) d = to;  // v >= N: dropped
        }
      }
      w.x = v;
      w.w = hop;
      *(reinterpret_cast<uint4*>(walks) + i) = w;
    }
    // rank among the row's walks of the same destination
    __syncwarp();
    const uint32_t peers = __match_any_sync(~0u, d);
    const uint32_t before = __popc(peers & ((1u << lane) - 1u));
    const bool leads = d != kNoDest && before == 0;
    if (leads) wcnt[warp * nb + d] = (uint8_t)__popc(peers);
    if (d != kNoDest) atomicMin(minhop + d, hop);
    __syncthreads();
    if (i < n) {
      uint32_t rank = before;
      if (d != kNoDest) {
        rank += total[d];
        for (uint32_t x = 0; x < warp; ++x) rank += wcnt[x * nb + d];
      }
      ps.dest[i] = d == kNoDest ? kNoDest : d | rank << 16;
    }
    __syncthreads();
    if (leads) {
      atomicAdd(total + d, (uint32_t)__popc(peers));
      wcnt[warp * nb + d] = 0;
    }
    if (++row == plan.rows || base + (uint64_t)row * kWalkThreads >= n) break;
    i += kWalkThreads;
    if (i < n) w = *(reinterpret_cast<const uint4*>(walks) + i);
  }
  __syncthreads();
  for (uint32_t b = threadIdx.x; b < nb; b += kWalkThreads) {
    ps.tile_hist[(uint64_t)b * plan.ntiles + blockIdx.x] = total[b];
    if (total[b]) atomicMin(ps.minhop + (size_t)b * kMinhopStride, minhop[b]);
  }
  if (st) atomicOr(status, st);
  if (SINK == GW_SINK_CLOSURE_COUNT && clos) atomicAdd(s.closure, (unsigned long long)clos);
}

__global__ void unpack_words_kernel(const uint64_t* __restrict__ words,
                                    const uint32_t* __restrict__ ids, uint64_t n,
                                    uint32_t block_base, gw_walk_rec* __restrict__ out,
                                    uint32_t* __restrict__ minhop) {
  uint32_t low = 0xffffffffu;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t wd = words[i];
    const uint32_t src = (uint32_t)(wd >> 40) & 0xffffffu;
    uint4 r;
    r.x = block_base + ((uint32_t)(wd >> 14) & 0x3ffffffu);
    r.y = ids ? ids[i] : src;
    r.z = src;
    r.w = (uint32_t)(wd & 0x3fffu);
    low = min(low, r.w);
    *(reinterpret_cast<uint4*>(out) + i) = r;
  }
  if (minhop) {  // the lowest hop of the block's walks (the launch's threads are whole warps)
    low = __reduce_min_sync(~0u, low);
    if ((threadIdx.x & 31) == 0 && low != 0xffffffffu) atomicMin(minhop, low);
  }
}

__global__ void unpack_pools_kernel(const uint64_t* __restrict__ words,
                                    const uint32_t* __restrict__ ids, uint64_t first, uint64_t n,
                                    const uint64_t* __restrict__ pool_offsets,
                                    const uint32_t* __restrict__ blocks, uint32_t nblocks,
                                    gw_walk_rec* __restrict__ out) {
  for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n;
       j += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t i = first + j;
    // pool of walk i: last p with pool_offsets[p] <= i
    uint32_t lo = 0, hi = nblocks;
    while (lo < hi) {
      const uint32_t mid = (lo + hi + 1) >> 1;
      if (__ldg(pool_offsets + mid) <= i) lo = mid;
      else hi = mid - 1;
    }
    const uint64_t wd = words[j];
    const uint32_t src = (uint32_t)(wd >> 40) & 0xffffffu;
    uint4 r;
    r.x = __ldg(blocks + lo) + ((uint32_t)(wd >> 14) & 0x3ffffffu);
    r.y = ids ? ids[j] : src;
    r.z = src;
    r.w = (uint32_t)(wd & 0x3fffu);
    *(reinterpret_cast<uint4*>(out) + j) = r;
  }
}

__global__ void pack_words_kernel(const gw_walk_rec* __restrict__ walks, uint64_t n,
                                  const uint32_t* __restrict__ blocks, uint32_t nblocks,
                                  uint64_t* __restrict__ words, uint32_t* __restrict__ wblock) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint4 w = *(reinterpret_cast<const uint4*>(walks) + i);
    const uint32_t p = find_block(blocks, nblocks, w.x);
    const uint32_t rel = p < nblocks ? w.x - __ldg(blocks + p) : w.x;
    words[i] = (((uint64_t)w.z & 0xffffffu) << 40) | (((uint64_t)rel & 0x3ffffffu) << 14) |
               ((uint64_t)w.w & 0x3fffu);
    if (wblock) wblock[i] = p;
  }
}

// Random-sector gather probe: each thread issues independent 4-byte loads at
// hashed positions of a buffer much larger than L2, so every load is its own
// 32-byte DRAM sector.  The sum is kept live through *sink.
__global__ void __launch_bounds__(256)
    gather_probe_kernel(const uint32_t* __restrict__ buf, uint64_t n_words, uint64_t loads,
                        unsigned long long* __restrict__ sink) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  uint32_t acc = 0;
  // sectors in the buffer, rounded down to a power of two (mask, no modulo)
  uint64_t nsect = 1;
  while (nsect * 2 <= n_words / 8) nsect *= 2;
  const uint32_t mask = (uint32_t)(nsect - 1);
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < loads; i += stride * 4) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint64_t j = i + u * stride;
      if (j < loads) {
        uint32_t h = (uint32_t)j * 0x9E3779B9u;
        h ^= h >> 15;
        h *= 0x85EBCA6Bu;
        h ^= h >> 13;
        acc += __ldg(buf + (uint64_t)(h & mask) * 8 + (j & 7));
      }
    }
  }
  if (acc == 0x9e3779b9u) atomicAdd(sink, 1ull);
}

// Random visit-counter updates alone: `ops` red.add of 1 at pseudo-random
// counters of c[0 .. mask] (mask + 1 a power of two), with the counters'
// evict_last policy, the same instruction the walk kernels count visits with.
__global__ void __launch_bounds__(256)
    red_probe_kernel(uint32_t* __restrict__ c, uint32_t mask, uint64_t ops) {
  const uint64_t pol = l2_policy(false, true);
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < ops; i += stride) {
    uint32_t h = (uint32_t)i * 0x9E3779B9u + (uint32_t)(i >> 32);
    h ^= h >> 16;
    h *= 0x7FEB352Du;
    h ^= h >> 15;
    red_add_u32(c + (h & mask), 1u, pol);
  }
}

int g_num_sms = 0;

int num_sms() {
  if (g_num_sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
    if (g_num_sms <= 0) g_num_sms = 148;
  }
  return g_num_sms;
}

template <typename K>
int ctas_per_sm(K kernel) {
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kWalkThreads, 0);
  return per_sm > 0 ? per_sm : 1;
}

int grid_of(int per_sm, uint64_t n) {
  const uint64_t full = (uint64_t)num_sms() * per_sm;
  const uint64_t need = (n + kWalkThreads - 1) / kWalkThreads;
  return (int)(need < full ? (need > 0 ? need : 1) : full);
}

// Whether n resident walks over g read its edge records.  A move along an edge
// record is one gather where the CSR takes two, but the records are four times
// the columns, and a jump over them waits for a bitmap word, the target's
// record and its edge in turn, in a warp whose other lanes wait for theirs.  So
// jumping walks read the CSR while its vertex records stay in the L2 beside the
// visit counters, and so do large sets of the rules that end at a failed test
// (us a launch, records in their shape / CSR; random starts, counts, the
// reference's jump probability where none is given):
//   jump: 4099 walks at R-MAT scale 14 15.4 / 9.8; 4 M at 22 833 / 702, with 40
//     edges a vertex (671 MB) 925 / 841; 4 M on uniform graphs of 12 edges a
//     vertex: 5.0 M vertices 1028 / 886, 6.0 M 1057 / 978, 7.0 M 1058 / 1038, 8.4 M
//     1078 / 1113.  Beyond, and with other jump probabilities, the CSR loses: R-MAT
//     23, 12 edges a vertex, probability 0.5: 561 / 671; 24 and 6 edges (511 MB):
//     16.8 M walks 3192 / 3903, 2044 / 3034 with 0.5.  It keeps the chain of hops
//     short for few walks: 24 and 6 edges 30,000 19.3 / 15.2 but 100,000 29.7 / 32.0;
//     23 and 16 edges 100,000 30.7 / 27.8, 300,000 76 / 71, 1 M 246 / 237 but 161 / 178
//     with 0.5.  One walk per vertex at 24 and 16 edges 3638 / 4210.
//   stop, uncapped: 1 M at 21 91 / 78 and 134 / 119; 4 M at 22 (301 MB) 336 / 308
//     and 456 / 416, at 23 389 / 398 and 501 / 508, at 24 and 2 edges (255 MB) 252 /
//     288 (stop); few walks 11.1 / 12.3 (4099 at 23): a chain of hops with two
//     gathers each;
//   PPR, restart: their walks go back to a source whose record they hold (PPR:
//     1 M at 20 148 / 162, 4 M at 22 560 / 656; restart: 127 / 122, 513 / 534).
template <int RULE>
bool walks_use_records(const GraphPlan& g, uint64_t n) {
  constexpr uint32_t kCachedVertices = (48u << 20) / 8;  // whose records take 48 MB
  if (!g.erec) return false;
  if (RULE == GW_RULE_JUMP) {
    const bool few = n < (g.nv <= 1u << 23 ? 1u << 18 : 1u << 16);
    return g.csr_bytes > g.csr_limit || (g.nv > kCachedVertices && !few);
  }
  return rule_returns<RULE>() || n < 1u << 19 || g.csr_bytes > g.csr_limit / 2 || g.nv > kCachedVertices;
}

// CTAs per SM of a resident launch that no autotuner shaped: all that fit,
// except where fewer requests in flight queue less at the DRAM: jumps over
// edge records (one walk per vertex at scale 24: 8 CTAs 4.02 ms, 6 3.81, 5 3.74,
// 4 3.80; at 23 1749, 1684, 1684, 1714 us; up to a jump probability of about 0.3:
// 23 and 12 edges a vertex 8 CTAs 803, 5 783 us with 0.25, 680 and 682 with 0.35,
// 528 and 561 with 0.5), and restarting walks that record
// paths beyond a third of the L2, whose rows then fill before they are written
// out (3 M at 22, 11 visits: 8 CTAs 352 us, 6 332; 2 M at 21, 20 visits: 1.08
// times; under 40 MB 0.94 to 1.04 times; stop walks' paths take 1.03 to 1.1
// times as long with 6, PPR's 0.92 to 1.1).  The PPR rule, whose walks end
// early, wants them all (24: 2.21 ms with 8, 2.83 with 5).
template <int RULE, int SINK>
int default_ctas_per_sm(bool records, uint64_t n, const WalkArgs& a) {
  if (RULE == GW_RULE_JUMP && records && a.thr <= 0x80000000u / 10 * 3) return 5;
  if (RULE == GW_RULE_RESTART && SINK == GW_SINK_PATH_RECORD && n * a.path_stride * 4 >= 40u << 20) return 6;
  return 1 << 16;
}

template <int RULE, int SINK, bool AGG>
WalkShape resident_shape(uint64_t n, const GraphPlan& g, const WalkArgs& a) {
  // a kernel's occupancy is asked for once: the call takes as long as a short launch
  static const int fit[2] = {ctas_per_sm(walk_resident_kernel<RULE, SINK, AGG, false>),
                             ctas_per_sm(walk_resident_kernel<RULE, SINK, AGG, true>)};
  WalkShape s;
  s.records = walks_use_records<RULE>(g, n);
  s.fit = fit[s.records];
  const int tuned = g.shapes ? g.shapes->ctas[RULE][SINK][s.records] : 0;
  s.ctas = std::min(s.fit, tuned > 0 ? tuned : default_ctas_per_sm<RULE, SINK>(s.records, n, a));
  return s;
}

template <int RULE, int SINK, bool AGG>
cudaError_t resident_dispatch(const gw_walk_rec* walks, uint64_t n, const GraphPlan& g,
                              const WalkArgs& a, const SinkView& s, uint32_t* status,
                              cudaStream_t stream, const cudaAccessPolicyWindow* window) {
  const WalkShape shape = resident_shape<RULE, SINK, AGG>(n, g, a);
  const int grid = grid_of(shape.ctas, n);
  auto k = shape.records ? walk_resident_kernel<RULE, SINK, AGG, true> : walk_resident_kernel<RULE, SINK, AGG, false>;
  if (!window) {
    k<<<grid, kWalkThreads, 0, stream>>>(walks, n, g, a, s, status);
    return cudaGetLastError();
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kWalkThreads);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeAccessPolicyWindow;
  attr[0].val.accessPolicyWindow = *window;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, walks, n, g, a, s, status);
}

template <int RULE, int SINK, bool AGG>
cudaError_t block_dispatch(gw_walk_rec* walks, uint64_t n, const GraphView& g,
                           const unsigned long long* beg_pos, const uint32_t* csr,
                           const WalkArgs& a, const SinkView& s, const uint32_t* blocks,
                           const PartitionPlan& plan, const PartitionScratch& ps, uint32_t* status,
                           cudaStream_t stream) {
  auto k = beg_pos ? walk_block_kernel<RULE, SINK, AGG, true> : walk_block_kernel<RULE, SINK, AGG, false>;
  const size_t nb = plan.nbuckets;
  const size_t smem = nb * (8 + kWalkThreads / 32) + (nb <= kStagedBlocks ? (nb + 1) * 4 : 0);
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  k<<<plan.ntiles, kWalkThreads, smem, stream>>>(walks, n, g, beg_pos, csr, a, s, blocks, plan, ps, status);
  return cudaGetLastError();
}

}  // namespace

// Dispatch a (rule, sink, aggregate) triple to its template instance.
#define GW_SINK_CASES(RULE, FN, ...)                                                   \
  switch (sink) {                                                                      \
    case GW_SINK_NONE: return FN<RULE, GW_SINK_NONE, false>(__VA_ARGS__);              \
    case GW_SINK_VERTEX_COUNT:                                                         \
      return agg ? FN<RULE, GW_SINK_VERTEX_COUNT, true>(__VA_ARGS__)                   \
                 : FN<RULE, GW_SINK_VERTEX_COUNT, false>(__VA_ARGS__);                 \
    case GW_SINK_PATH_RECORD: return FN<RULE, GW_SINK_PATH_RECORD, false>(__VA_ARGS__); \
    case GW_SINK_CLOSURE_COUNT: return FN<RULE, GW_SINK_CLOSURE_COUNT, false>(__VA_ARGS__); \
  }
#define GW_RULE_CASES(FN, ...)                                         \
  switch (rule) {                                                      \
    case GW_RULE_JUMP: GW_SINK_CASES(GW_RULE_JUMP, FN, __VA_ARGS__) break;       \
    case GW_RULE_STOP: GW_SINK_CASES(GW_RULE_STOP, FN, __VA_ARGS__) break;       \
    case GW_RULE_PROB: GW_SINK_CASES(GW_RULE_PROB, FN, __VA_ARGS__) break;       \
    case GW_RULE_RESTART: GW_SINK_CASES(GW_RULE_RESTART, FN, __VA_ARGS__) break; \
    case GW_RULE_PPR: GW_SINK_CASES(GW_RULE_PPR, FN, __VA_ARGS__) break;         \
  }

cudaError_t launch_walk_resident(int rule, int sink, bool agg, const gw_walk_rec* walks, uint64_t n,
                                 const GraphPlan& g, const WalkArgs& a, const SinkView& s,
                                 uint32_t* status, cudaStream_t stream,
                                 const cudaAccessPolicyWindow* window) {
  if (n == 0) return cudaSuccess;
  GW_RULE_CASES(resident_dispatch, walks, n, g, a, s, status, stream, window)
  return cudaErrorInvalidValue;
}

WalkShape walk_resident_shape(int rule, int sink, bool agg, uint64_t n, const GraphPlan& g, const WalkArgs& a) {
  GW_RULE_CASES(resident_shape, n, g, a)
  return WalkShape{false, 1, 1};
}

cudaError_t launch_walk_block(int rule, int sink, bool agg, gw_walk_rec* walks, uint64_t n,
                              const GraphView& g, const unsigned long long* beg_pos,
                              const uint32_t* csr, const WalkArgs& a, const SinkView& s,
                              const uint32_t* blocks, const PartitionPlan& plan, const PartitionScratch& ps,
                              uint32_t* status, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  if (sink == GW_SINK_PATH_RECORD) return cudaErrorInvalidValue;
  GW_RULE_CASES(block_dispatch, walks, n, g, beg_pos, csr, a, s, blocks, plan, ps, status, stream)
  return cudaErrorInvalidValue;
}

static int elementwise_grid(uint64_t n) {
  const uint64_t need = (n + 255) / 256;
  const uint64_t cap = (uint64_t)num_sms() * 16;
  return (int)(need < cap ? (need ? need : 1) : cap);
}

cudaError_t launch_unpack_words(const uint64_t* words, const uint32_t* ids, uint64_t n,
                                uint32_t block_base, gw_walk_rec* out, cudaStream_t stream, uint32_t* minhop) {
  if (n == 0) return cudaSuccess;
  unpack_words_kernel<<<elementwise_grid(n), 256, 0, stream>>>(words, ids, n, block_base, out, minhop);
  return cudaGetLastError();
}

cudaError_t launch_unpack_pools(const uint64_t* words, const uint32_t* ids, uint64_t first,
                                uint64_t n, const uint64_t* pool_offsets, const uint32_t* blocks,
                                uint32_t nblocks, gw_walk_rec* out, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  unpack_pools_kernel<<<elementwise_grid(n), 256, 0, stream>>>(words, ids, first, n, pool_offsets,
                                                               blocks, nblocks, out);
  return cudaGetLastError();
}

cudaError_t launch_pack_words(const gw_walk_rec* walks, uint64_t n, const uint32_t* blocks,
                              uint32_t nblocks, uint64_t* words, uint32_t* wblock,
                              cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  pack_words_kernel<<<elementwise_grid(n), 256, 0, stream>>>(walks, n, blocks, nblocks, words,
                                                             wblock);
  return cudaGetLastError();
}

cudaError_t launch_build_erec(const uint32_t* colidx, const unsigned long long* vrec, uint64_t ne, uint32_t nv,
                              ulonglong2* erec, cudaStream_t stream) {
  if (ne == 0) return cudaSuccess;
  build_erec_kernel<<<elementwise_grid(ne), 256, 0, stream>>>(colidx, vrec, ne, nv, erec);
  return cudaGetLastError();
}

cudaError_t launch_gather_probe(const uint32_t* buf, uint64_t n_words, uint64_t loads,
                                unsigned long long* sink, cudaStream_t stream) {
  const int grid = num_sms() * 8;
  gather_probe_kernel<<<grid, 256, 0, stream>>>(buf, n_words, loads, sink);
  return cudaGetLastError();
}

cudaError_t launch_red_probe(uint32_t* counters, uint32_t mask, uint64_t ops, cudaStream_t stream) {
  red_probe_kernel<<<num_sms() * 8, 256, 0, stream>>>(counters, mask, ops);
  return cudaGetLastError();
}

}  // namespace gw
