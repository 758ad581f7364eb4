// gw_partition.cu -- stable on-device partition of walks by destination block.
//
// Replaces WalkManager::moveWalk + WalkBuffer::push_back + the per-block
// pools (src/walks/walk.hpp:93-137, src/walks/walkbuffer.hpp:32-39).  The
// reference appends each exiting walk to a per-(thread, block) buffer, so the
// order inside a pool depends on the thread schedule; here the order is
// defined: a destination pool receives the walks of a superstep in input
// order (a stable counting sort over one digit = the destination block).
//
// The walk kernel (gw_walk.cu) leaves each walk's destination and its rank in
// its tile, and each tile's count per destination.  What remains is one scan
// of the tile counts, a CTA per destination, and one elementwise scatter.  The
// scan also places every destination's walks in its pool from a table the
// device keeps, so the scatter is queued right behind it and the host learns
// the totals (mapped memory) while the scatter runs, not before it.
//
// Measured at R-MAT scale 22, 33 blocks, 126 k walks per superstep (ncu, one
// launch each): histogram 10.4, scan 7.7, totals 4.6, pool pointers read over
// the host link 4.6 and scatter 7.4 us, five launches and a host wait in
// their middle, when the walk kernel left only the destinations.
#include <algorithm>

#include "gw_internal.h"

namespace gw {

namespace {

constexpr int kScanThreads = 512;
constexpr int kScanWarps = kScanThreads / 32;

__device__ __forceinline__ unsigned long long device_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// One CTA per bucket: exclusive scan of its row of tile counts, in place.
__global__ void __launch_bounds__(kScanThreads)
    partition_scan_kernel(PartitionPlan plan, PartitionScratch ps, uint32_t* totals, uint32_t* minhop_out,
                          PoolTable pools, uint32_t block, uint64_t* moved, uint16_t seq) {
  __shared__ uint32_t wsum[2][kScanWarps];  // alternating: one barrier per step
  const uint32_t b = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  let_next_start();
  wait_for_previous();
  if (ps.clock && b == 0 && threadIdx.x == 0) {
    const unsigned long long t = device_ns(), end = ps.clock[kScatterEnd];
    if (end > ps.clock[kPartStart]) ps.clock[kPartSum] += end - ps.clock[kPartStart];  // the superstep before
    ps.clock[kWalkSum] += t - ps.clock[kWalkStart];
    ps.clock[kPartStart] = t;
  }
  uint32_t* const row = ps.tile_hist + (uint64_t)b * plan.ntiles;
  uint32_t carry = 0;
  for (uint32_t t0 = 0, step = 0; t0 < plan.ntiles; t0 += kScanThreads, ++step) {
    const uint32_t t = t0 + threadIdx.x;
    const uint32_t c = t < plan.ntiles ? row[t] : 0u;
    uint32_t incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(~0u, incl, o);
      if (lane >= (uint32_t)o) incl += y;
    }
    uint32_t* const ws = wsum[step & 1];
    if (lane == 31) ws[warp] = incl;
    __syncthreads();
    // every warp scans the warp sums itself
    const uint32_t x = lane < kScanWarps ? ws[lane] : 0u;
    uint32_t y = x;
#pragma unroll
    for (int o = 1; o < kScanWarps; o <<= 1) {
      const uint32_t z = __shfl_up_sync(~0u, y, o);
      if (lane >= (uint32_t)o) y += z;
    }
    const uint32_t below = __shfl_sync(~0u, y - x, warp);
    if (t < plan.ntiles) row[t] = carry + below + incl - c;
    carry += __shfl_sync(~0u, y, kScanWarps - 1);
  }
  if (threadIdx.x != 0) return;
  uint32_t* const minhop = ps.minhop + (size_t)b * kMinhopStride;
  const uint32_t low = *minhop;
  *minhop = 0xffffffffu;  // for the next superstep
  if (!moved) {
    totals[b] = carry;
    minhop_out[b] = low;
    return;
  }
  *reinterpret_cast<volatile uint64_t*>(moved + b) = moved_word(carry, low, seq);
  const uint64_t held = b == block ? 0 : pools.n[b];
  pools.place[b] = held;
  pools.n[b] = held + carry;
  if (held + carry > pools.cap[b]) atomicOr(pools.full, 1u);
}

__global__ void fetch_pools_kernel(const uint64_t* src, PoolTable pools, uint32_t nb) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nb; i += gridDim.x * blockDim.x) {
    pools.ptr[i] = reinterpret_cast<gw_walk_rec*>(src[i]);
    pools.n[i] = src[nb + i];
    pools.cap[i] = src[2 * nb + i];
    pools.place[i] = src[3 * nb + i];
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *pools.full = 0;
}

// One walk per thread: 16 bytes in, 16 out, and 4 bytes of destination; its
// tile's offset, its pool's pointer and place are cache hits.
__global__ void __launch_bounds__(256)
    partition_scatter_kernel(const gw_walk_rec* walks, uint64_t n, PartitionPlan plan, PartitionScratch ps,
                             gw_walk_rec* const* ptr, const uint64_t* place, const uint32_t* full) {
  wait_for_previous();
  if (full && *full) return;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t x = ps.dest[i];
    if (x == kNoDest) continue;
    const uint32_t d = x & 0xffffu, tile = (uint32_t)(i / plan.tile());
    const uint4 w = __ldcg(reinterpret_cast<const uint4*>(walks) + i);
    const uint64_t pos = place[d] + ps.tile_hist[(uint64_t)d * plan.ntiles + tile] + (x >> 16);
    *(reinterpret_cast<uint4*>(ptr[d]) + pos) = w;
  }
  if (ps.clock && threadIdx.x == 0) atomicMax(ps.clock + kScatterEnd, device_ns());
}

}  // namespace

PartitionPlan partition_plan(uint64_t n, uint32_t nbuckets) {
  // One row of 256 walks per tile while the tiles fit one wave of eight CTAs
  // per SM (300 k walks): fewest walks behind a barrier.  Above it, tiles of
  // more rows keep the tile counts (4 bytes per destination and tile, written,
  // scanned and read) small beside the walks.
  constexpr uint64_t kWave = 148 * 8;
  PartitionPlan p;
  p.nbuckets = nbuckets;
  const uint64_t rows = (n + kWave * kWalkThreads - 1) / (kWave * kWalkThreads);
  p.rows = (uint32_t)std::min<uint64_t>(std::max<uint64_t>(rows, 1), kMaxRows);
  p.ntiles = (uint32_t)((n + p.tile() - 1) / p.tile());
  return p;
}

cudaError_t launch_partition_scan(const PartitionPlan& plan, const PartitionScratch& ps, uint32_t* totals,
                                  uint32_t* minhop_out, cudaStream_t stream) {
  if (plan.nbuckets == 0) return cudaSuccess;
  return launch_dependent(partition_scan_kernel, plan.nbuckets, kScanThreads, 0, stream, plan, ps, totals, minhop_out,
                          PoolTable{}, 0u, (uint64_t*)nullptr, (uint16_t)0);
}

cudaError_t launch_partition_scan(const PartitionPlan& plan, const PartitionScratch& ps, const PoolTable& pools,
                                  uint32_t block, uint64_t* moved, uint16_t seq, cudaStream_t stream) {
  if (plan.nbuckets == 0) return cudaSuccess;
  return launch_dependent(partition_scan_kernel, plan.nbuckets, kScanThreads, 0, stream, plan, ps, (uint32_t*)nullptr,
                          (uint32_t*)nullptr, pools, block, moved, seq);
}

cudaError_t launch_fetch_pools(const uint64_t* src, const PoolTable& pools, uint32_t nbuckets, cudaStream_t stream) {
  if (nbuckets == 0) return cudaSuccess;
  fetch_pools_kernel<<<std::min<uint32_t>((nbuckets + 255) / 256, 64), 256, 0, stream>>>(src, pools, nbuckets);
  return cudaGetLastError();
}

cudaError_t launch_partition_scatter(const gw_walk_rec* walks, uint64_t n, const PartitionPlan& plan,
                                     const PartitionScratch& ps, gw_walk_rec* const* ptr, const uint64_t* place,
                                     const uint32_t* full, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  const uint64_t ctas = std::min<uint64_t>((n + 255) / 256, 1u << 20);
  return launch_dependent(partition_scatter_kernel, (unsigned)ctas, 256, 0, stream, walks, n, plan, ps, ptr, place,
                          full);
}

}  // namespace gw
