// gw_internal.h -- host-side declarations shared by the library's sources.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <string>
#include <vector>

#include "../../include/graphwalker_b200.h"
#include "gw_device.cuh"

namespace gw {

constexpr int kWalkThreads = 256;

// Device status bits (OR-ed into the context's status word by kernels).
constexpr uint32_t kStBounds = 1u;    // vertex id >= nvertices met
constexpr uint32_t kStOverflow = 2u;  // path stride / table capacity exceeded
constexpr uint32_t kStHops = 4u;      // uncapped walk exceeded max_hops

// L2 hints the walk kernels use when the caller asks for the default: column
// loads are evicted first and the visit counters kept (measured on B200 at
// R-MAT scale 24: 1.10x alone, 1.41x with the counters' persisting window).
constexpr uint32_t kDefaultHints = kHintColumnsEvictFirst | kHintCountsEvictLast;

// ---- walk kernels (gw_walk.cu) ----
// window (may be NULL): an L2 access policy window attached to the launch.
cudaError_t launch_walk_resident(int rule, int sink, bool agg, const gw_walk_rec* walks, uint64_t n,
                                 const GraphPlan& g, const WalkArgs& a, const SinkView& s,
                                 uint32_t* status, cudaStream_t stream,
                                 const cudaAccessPolicyWindow* window = nullptr);
// The layout that launch takes for n walks, its CTAs per SM, and the most that fit.
struct WalkShape {
  bool records;
  int ctas, fit;
};
WalkShape walk_resident_shape(int rule, int sink, bool agg, uint64_t n, const GraphPlan& g, const WalkArgs& a);

// ---- codec kernels (gw_walk.cu) ----
// minhop (may be NULL): atomicMin of the walks' lowest hop.
cudaError_t launch_unpack_words(const uint64_t* words, const uint32_t* ids, uint64_t n,
                                uint32_t block_base, gw_walk_rec* out, cudaStream_t stream,
                                uint32_t* minhop = nullptr);
// Words of several pools laid end to end: pool p = [pool_offsets[p], pool_offsets[p+1]).
cudaError_t launch_unpack_pools(const uint64_t* words, const uint32_t* ids, uint64_t first,
                                uint64_t n, const uint64_t* pool_offsets, const uint32_t* blocks,
                                uint32_t nblocks, gw_walk_rec* out, cudaStream_t stream);
cudaError_t launch_pack_words(const gw_walk_rec* walks, uint64_t n, const uint32_t* blocks,
                              uint32_t nblocks, uint64_t* words, uint32_t* wblock,
                              cudaStream_t stream);
// SimRank meeting counts meet[q * L + l] of nq queries: query q compares the
// R x L path rows at element offset rows[2q] of a with rows[2q + 1] of b
// (rows NULL: one query at offset 0 of both) (gw_simrank.cu).
cudaError_t launch_simrank_meet(const uint32_t* a, const uint32_t* b, const unsigned long long* rows, uint32_t nq,
                                uint32_t R, uint32_t L, unsigned long long* meet, cudaStream_t stream);
// Walk records of SimRank's placement: walk k * R + i = replica i of verts[k].
cudaError_t launch_simrank_walks(const uint32_t* verts, uint32_t nverts, uint32_t R, uint32_t L, gw_walk_rec* out,
                                 cudaStream_t stream);
// erec[e] = (packed record of colidx[e], colidx[e]) for e < ne (gw_walk.cu).
cudaError_t launch_build_erec(const uint32_t* colidx, const unsigned long long* vrec, uint64_t ne, uint32_t nv,
                              ulonglong2* erec, cudaStream_t stream);

// ---- graph kernels (gw_graph.cu) ----
// Bytes of the vertex-record buffer: nv packed records, then the out-edge
// bitmap (one bit per vertex, in 32-bit words).
inline size_t vrec_bytes(uint32_t nv) { return (size_t)nv * 8 + (((size_t)nv + 31) / 32) * 4; }
// Fills the packed records and the out-edge bitmap (vrec_bytes(nv) bytes at vrec).
cudaError_t launch_build_vrec(const unsigned long long* rowptr, uint32_t nv,
                              unsigned long long* vrec, cudaStream_t stream);
// rowptr[nv + 1] and colidx[n] of edge keys (source << 32 | target) sorted by
// source (gw_graph.cu).
cudaError_t launch_rowptr_from_sorted(const unsigned long long* keys, uint64_t n, uint32_t nv,
                                      unsigned long long* rowptr, uint32_t* colidx, cudaStream_t stream);
// R-MAT CSR on the device.  On success *rowptr_out / *colidx_out are new
// device allocations (cudaMalloc) and *nedges the kept edge count.
cudaError_t rmat_build_csr(uint32_t scale, uint64_t nedges_raw, uint64_t seed, uint32_t ta,
                           uint32_t tab, uint32_t tabc, unsigned long long** rowptr_out,
                           uint32_t** colidx_out, uint64_t* nedges, cudaStream_t stream);

// Launches k so that its CTAs may start while the kernel before it on the
// stream drains (programmatic dependent launch): k must call
// wait_for_previous() before it touches anything an earlier kernel writes or
// reads.  What an earlier kernel of the stream writes is read with ordinary,
// __ldcg or relaxed loads: the read-only path (__ldg, ld.global.nc, and so
// `const T* __restrict__` parameters) wants data that no one writes from the
// kernel's start on, and this kernel starts before its predecessors end.
template <typename... P, typename... A>
cudaError_t launch_dependent(void (*k)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t stream,
                             A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, P(args)...);
}

// ---- block supersteps: walk + stable partition (gw_walk.cu, gw_partition.cu) ----
constexpr uint32_t kNoDest = 0xffffffffu;    // dest[] of a walk that ended
constexpr uint32_t kStagedBlocks = 2048;     // block ranges up to here are searched in shared memory
constexpr uint32_t kMaxRows = 64;            // rows of a tile: ranks stay below 2^16
constexpr uint32_t kMaxBuckets = 8000;       // shared memory of the walk kernel: 16 bytes per destination

// The walks of a superstep in tiles of `rows` x kWalkThreads; one CTA walks a tile.
struct PartitionPlan {
  uint32_t nbuckets = 0;  // destination blocks
  uint32_t ntiles = 0;
  uint32_t rows = 1;
  __host__ __device__ uint32_t tile() const { return rows * kWalkThreads; }
};
PartitionPlan partition_plan(uint64_t n, uint32_t nbuckets);

// Every tile adds its lowest hops to the buckets' by atomics, so each bucket's
// has a 128-byte line of its own: side by side, what they cost went by the
// address the allocator gave the array (R-MAT scale 20, 261 blocks, 4000 walks a
// superstep: 12.4 or 16.3 us of partition a superstep, 7.7 so; in 32-byte sectors
// 8.8).
constexpr uint32_t kMinhopStride = 32;

// Device arrays a superstep's kernels hand on.
struct PartitionScratch {
  uint32_t* dest;       // per walk: destination | rank in the tile << 16, or kNoDest
  uint32_t* tile_hist;  // [bucket * ntiles + tile]: walk counts, then their exclusive scan per bucket
  uint32_t* minhop;     // per bucket, kMinhopStride apart: lowest hop of the walks that move there (0xffffffff = none)
  unsigned long long* clock;  // NULL, or the superstep clock, kClockWords of device ns
};
// The superstep clock: when the walk and the partition of the last superstep
// started and when its scatter ended (the latest CTA's stamp), and what the
// supersteps before it took in sum, walking and partitioning.
enum : uint32_t { kWalkStart, kPartStart, kScatterEnd, kWalkSum, kPartSum, kClockWords };

// The device pools a superstep's walks move to, one entry per block.  The scan
// places the new walks behind the n held, advances n and empties the block
// that ran.  When a pool is too small for its new walks it sets *full: the
// scatter then does nothing, and the host grows the pools, uploads the table
// (launch_fetch_pools) and launches the scatter again.
struct PoolTable {
  // Entries from one array to the next: whole 128-byte lines, so that no line
  // holds both what the scan reads and what it writes for the scatter.
  static size_t stride(uint32_t nbuckets) { return ((size_t)nbuckets + 15) / 16 * 16; }
  gw_walk_rec** ptr;
  uint64_t* n;      // records held
  uint64_t* cap;    // records the pool has room for
  uint64_t* place;  // where the scatter puts a bucket's first walk
  uint32_t* full;   // some pool is too small: the scatter does nothing
};

// What the scan tells the host about a bucket, one 64-bit word in mapped
// pinned memory written by one store: total | min(minimum hop, 0xffff) << 32 |
// seq << 48.  The host polls every bucket's word for the superstep's seq, so
// the scan needs no fence and no last CTA before its kernel can end.
__host__ __device__ inline uint64_t moved_word(uint32_t total, uint32_t minhop, uint16_t seq) {
  return total | (uint64_t)(minhop < 0xffffu ? minhop : 0xffffu) << 32 | (uint64_t)seq << 48;
}

// Blocked-mode superstep: advances the n walks of one block while they stay
// inside [a.lo, a.hi), writes them back in place, and leaves ps.dest,
// ps.tile_hist (one column per tile) and ps.minhop.  beg_pos/csr non-null =
// block slice.
cudaError_t launch_walk_block(int rule, int sink, bool agg, gw_walk_rec* walks, uint64_t n,
                              const GraphView& g, const unsigned long long* beg_pos,
                              const uint32_t* csr, const WalkArgs& a, const SinkView& s,
                              const uint32_t* blocks, const PartitionPlan& plan, const PartitionScratch& ps,
                              uint32_t* status, cudaStream_t stream);
// Exclusive scan of every bucket's tile counts in place.  The totals and the
// minimum hops (reset for the next superstep) go to totals[b] and
// minhop_out[b], or, with a pool table, to moved[b] (moved_word), and the
// buckets are placed in their pools (`block` is the one that ran).
cudaError_t launch_partition_scan(const PartitionPlan& plan, const PartitionScratch& ps, uint32_t* totals,
                                  uint32_t* minhop_out, cudaStream_t stream);
cudaError_t launch_partition_scan(const PartitionPlan& plan, const PartitionScratch& ps, const PoolTable& pools,
                                  uint32_t block, uint64_t* moved, uint16_t seq, cudaStream_t stream);
// Copies the host's table (src: nbuckets entries each of ptr, n, cap, place)
// into `pools` and clears *full, by a kernel: src may be mapped pinned host
// memory written by the host before the launch.  Unlike an async
// host-to-device copy this does not queue behind large block copies on the
// copy engine.
cudaError_t launch_fetch_pools(const uint64_t* src, const PoolTable& pools, uint32_t nbuckets, cudaStream_t stream);
// Stable scatter: walk i with destination d and rank r lands at
// ptr[d][place[d] + tile_hist[d][its tile] + r]; does nothing when *full
// (full NULL: never).  Ended walks are not written.
cudaError_t launch_partition_scatter(const gw_walk_rec* walks, uint64_t n, const PartitionPlan& plan,
                                     const PartitionScratch& ps, gw_walk_rec* const* ptr, const uint64_t* place,
                                     const uint32_t* full, cudaStream_t stream);

// ---- measurement ----
cudaError_t launch_gather_probe(const uint32_t* buf, uint64_t n_words, uint64_t loads,
                                unsigned long long* sink, cudaStream_t stream);
// `ops` red.add of 1 at pseudo-random counters of counters[0 .. mask].
cudaError_t launch_red_probe(uint32_t* counters, uint32_t mask, uint64_t ops, cudaStream_t stream);

}  // namespace gw
