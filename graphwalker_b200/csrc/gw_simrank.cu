// gw_simrank.cu -- SimRank's meeting reduction on the device: the triple loop
// of SimRank::computeResult (apps/simrank.cpp:71-84).  For every pair (i, j)
// of the R walks from a and the R walks from b, the first position l < L at
// which both walks stand on the same vertex (0xFFFFFFFF = no visit never
// matches); meet[l] counts the pairs.  The app's estimate is
// sum_l meet[l] * 0.8^l / R^2.
//
// The host loop is O(R^2 L).  Two kernels do it here, both exact:
//
//  * simrank_pairs_kernel compares every pair: a CTA takes a 64 x 64 tile of
//    pairs, the two tiles' visits staged in shared memory 32 positions at a
//    time; each thread owns a 4 x 4 block of pairs and keeps their "met" flags
//    in a 16-bit mask.  Integer-ALU bound (87 %): 1647 us for 512 queries of
//    R = 1000, L = 11 on a scale-20 graph.
//  * simrank_join_kernel: few pairs ever stand on the same vertex (about 90 of
//    a million per position there), so a CTA joins a tile of a's walks with a
//    tile of b's by hashing, O(R) work a position, and only a pair that
//    matches is checked against its earlier positions.  A pair counts at its
//    first match only, so the counts are the loop's, whatever the order.
//    251 us for the same queries; bound by issue slots and the latency of
//    two barriers and a few shared-memory round trips per position.
//
// The join has 30 us of such latency even for one query, and its chains grow
// when walks coincide, so small batches keep comparing pairs (kPairWork).  The
// grid's z dimension runs over queries: query q compares the R walks at row
// offset rows[2q] of `a` with those at rows[2q + 1] of `b`.
#include <algorithm>

#include "gw_internal.h"

namespace gw {

namespace {

constexpr int kPairTile = 64;      // walks per tile side
constexpr int kPairChunk = 32;     // positions staged at a time
constexpr int kPairThreads = 256;  // 16 x 16 threads, 4 x 4 pairs each

__global__ void __launch_bounds__(kPairThreads)
    simrank_pairs_kernel(const uint32_t* __restrict__ a0, const uint32_t* __restrict__ b0,
                        const unsigned long long* __restrict__ rows, uint32_t q0, uint32_t R, uint32_t L,
                        unsigned long long* __restrict__ meet0) {
  __shared__ uint32_t sa[kPairChunk][kPairTile + 1];
  __shared__ uint32_t sb[kPairChunk][kPairTile + 1];
  __shared__ uint32_t hist[kPairChunk];
  const uint32_t q = q0 + blockIdx.z;
  const uint32_t* __restrict__ a = a0 + (rows ? rows[2 * (size_t)q] : 0ull);
  const uint32_t* __restrict__ b = b0 + (rows ? rows[2 * (size_t)q + 1] : 0ull);
  unsigned long long* __restrict__ meet = meet0 + (size_t)q * L;
  const uint32_t i0 = blockIdx.y * kPairTile, j0 = blockIdx.x * kPairTile;
  const uint32_t tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  uint32_t met = 0;  // bit u * 4 + w: pair (i0 + ty + 16u, j0 + tx + 16w) has met
  for (uint32_t l0 = 0; l0 < L; l0 += kPairChunk) {
    __syncthreads();
    for (uint32_t x = threadIdx.x; x < kPairTile * kPairChunk; x += kPairThreads) {
      const uint32_t r = x / kPairChunk, c = x % kPairChunk;  // walk r of the tile, position l0 + c
      const bool in_l = l0 + c < L;
      sa[c][r] = in_l && i0 + r < R ? __ldg(a + (size_t)(i0 + r) * L + l0 + c) : 0xffffffffu;
      sb[c][r] = in_l && j0 + r < R ? __ldg(b + (size_t)(j0 + r) * L + l0 + c) : 0xffffffffu;
    }
    if (threadIdx.x < kPairChunk) hist[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t lend = L - l0 < (uint32_t)kPairChunk ? L - l0 : (uint32_t)kPairChunk;
    for (uint32_t c = 0; c < lend && met != 0xffffu; ++c) {
      uint32_t va[4], vb[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        va[u] = sa[c][ty + 16 * u];
        vb[u] = sb[c][tx + 16 * u];
      }
      uint32_t now = 0;
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int w = 0; w < 4; ++w)
          now |= (va[u] == vb[w] && va[u] != 0xffffffffu ? 1u : 0u) << (u * 4 + w);
      now &= ~met;
      if (now) {
        atomicAdd(&hist[c], (uint32_t)__popc(now));
        met |= now;
      }
    }
    __syncthreads();
    if (threadIdx.x < lend && hist[threadIdx.x]) atomicAdd(meet + l0 + threadIdx.x, (unsigned long long)hist[threadIdx.x]);
  }
}

constexpr uint32_t kSrPairs = 512;      // matching pairs listed per position
constexpr uint32_t kNoVisit = 0xffffffffu;
constexpr uint32_t kNoWalk = 0xffffffffu;

constexpr uint32_t kSrChunk = 12;  // positions staged at a time

// LOG: a tile is 2^LOG walks of each side, one of each per thread.
template <int LOG>
__global__ void __launch_bounds__(1 << LOG)
    simrank_join_kernel(const uint32_t* __restrict__ a0, const uint32_t* __restrict__ b0,
                        const unsigned long long* __restrict__ rows, uint32_t q0, uint32_t R, uint32_t L,
                        unsigned long long* __restrict__ meet0) {
  constexpr uint32_t kSrTile = 1 << LOG, kSrSlots = 2 * kSrTile;  // tables at most half full
  auto sr_slot = [](uint32_t v) { return (v * 0x9E3779B1u) >> (31 - LOG); };
  extern __shared__ uint32_t staged[];
  uint32_t(*const sa)[kSrTile + 1] = reinterpret_cast<uint32_t(*)[kSrTile + 1]>(staged);
  uint32_t(*const sb)[kSrTile + 1] = sa + kSrChunk;
  // Two tables, one cleared while the other is looked up.  A slot holds a
  // vertex (key; kNoVisit = free) and the walk entered last under it (head);
  // next[walk] is the walk entered before it.  Half of a position's walks can
  // stand on one vertex (the source they return to), so heads are exchanged,
  // which never retries.
  __shared__ uint32_t key[2][kSrSlots];
  __shared__ uint32_t head[2][kSrSlots];
  __shared__ uint32_t next[kSrTile];
  __shared__ uint32_t pairs[2][kSrPairs];  // a position's matches: walk of a << 16 | walk of b
  __shared__ uint32_t npairs[2];
  __shared__ uint32_t met;  // pairs of the tile that have met
  const uint32_t q = q0 + blockIdx.z, x = threadIdx.x;
  const uint32_t i0 = blockIdx.y * kSrTile, j0 = blockIdx.x * kSrTile;
  const uint32_t na = min(R - i0, (uint32_t)kSrTile), nb = min(R - j0, (uint32_t)kSrTile);
  const uint32_t* __restrict__ a = a0 + (rows ? rows[2 * (size_t)q] : 0ull) + (size_t)i0 * L;
  const uint32_t* __restrict__ b = b0 + (rows ? rows[2 * (size_t)q + 1] : 0ull) + (size_t)j0 * L;
  unsigned long long* __restrict__ meet = meet0 + (size_t)q * L;
  for (uint32_t s = x; s < 2 * kSrSlots; s += kSrTile) {
    key[0][s] = kNoVisit;  // both tables
    head[0][s] = kNoWalk;
  }
  if (x == 0) met = npairs[0] = npairs[1] = 0;
  uint32_t l0 = 0;  // first position staged
  // whether walks i and j shared no vertex at a position before l
  auto first_meeting = [&](uint32_t i, uint32_t j, uint32_t l) {
    uint32_t k = 0;
    for (; k < l0 && k < l; ++k) {
      const uint32_t p = __ldg(a + (size_t)i * L + k);
      if (p == __ldg(b + (size_t)j * L + k) && p != kNoVisit) return false;
    }
    for (; k < l; ++k) {
      const uint32_t p = sa[k - l0][i];
      if (p == sb[k - l0][j] && p != kNoVisit) return false;
    }
    return true;
  };
  uint32_t n = 0;  // pairs this thread found to meet first at the position before
  for (uint32_t l = 0;; ++l) {
    const uint32_t t = l & 1, c = l % kSrChunk;
    if (c == 0 && l < L) {
      const uint32_t w = min(L - l, (uint32_t)kSrChunk);  // rows of a tile lie one behind the other
      uint32_t r = x / w, z = x - r * w;
      const uint32_t dr = kSrTile / w, dz = kSrTile - dr * w;
      for (uint32_t y = 0; y < w; ++y) {
        sa[z][r] = r < na ? __ldg(a + (size_t)r * L + l + z) : kNoVisit;
        sb[z][r] = r < nb ? __ldg(b + (size_t)r * L + l + z) : kNoVisit;
        r += dr;
        z += dz;
        if (z >= w) {
          z -= w;
          ++r;
        }
      }
      l0 = l;
      __syncthreads();
    }
    // enter b's walks of this position; count the matches of the one before
    if (l < L) {
      const uint32_t v = sb[c][x];
      if (v != kNoVisit) {
        uint32_t s = sr_slot(v);
        for (;;) {
          uint32_t k = *reinterpret_cast<volatile uint32_t*>(&key[t][s]);
          if (k == kNoVisit) k = atomicCAS(&key[t][s], kNoVisit, v);
          if (k == kNoVisit || k == v) break;
          s = (s + 1) & (kSrSlots - 1);
        }
        next[x] = atomicExch(&head[t][s], x);
      }
    }
    if (l > 0) {
      const uint32_t listed = min(npairs[t ^ 1], kSrPairs);
      for (uint32_t y = x; y < listed; y += kSrTile) {
        const uint32_t p = pairs[t ^ 1][y];
        n += first_meeting(p >> 16, p & 0xffffu, l - 1) ? 1u : 0u;
      }
      n = __reduce_add_sync(~0u, n);
      if ((x & 31) == 0 && n) {
        atomicAdd(meet + l - 1, (unsigned long long)n);
        atomicAdd(&met, n);
      }
      n = 0;
    }
    __syncthreads();
    if (l == L || met == na * nb) break;  // met changes only after the next barrier
    // look a's walks up; clear the other table and the list just counted
    if (x == 0) npairs[t ^ 1] = 0;
    const uint32_t v = sa[c][x];
    if (v != kNoVisit) {
      uint32_t s = sr_slot(v), k;
      while ((k = key[t][s]) != v && k != kNoVisit) s = (s + 1) & (kSrSlots - 1);
      // Matches are listed and checked one per thread: checked here, a lane's
      // chain would hold its warp for one check after another.  What the list
      // has no room for is checked here.
      for (uint32_t j = k == v ? head[t][s] : kNoWalk; j != kNoWalk; j = next[j]) {
        const uint32_t y = atomicAdd(&npairs[t], 1u);
        if (y < kSrPairs) pairs[t][y] = x << 16 | j;
        else n += first_meeting(x, j, l) ? 1u : 0u;
      }
    }
    for (uint32_t s = x; s < kSrSlots; s += kSrTile) {
      key[t ^ 1][s] = kNoVisit;
      head[t ^ 1][s] = kNoWalk;
    }
    __syncthreads();
  }
}

// The app's placement (simrank.cpp:30-57): replica i of vertex v starts at v
// with hop i*L, keyed on v; walk k * R + i is replica i of verts[k].
__global__ void simrank_walks_kernel(const uint32_t* __restrict__ verts, uint64_t n, uint32_t R, uint32_t L,
                                     gw_walk_rec* __restrict__ out) {
  for (uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; w < n; w += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t v = __ldg(verts + w / R), i = (uint32_t)(w % R);
    reinterpret_cast<uint4*>(out)[w] = make_uint4(v, v, v, i * L);
  }
}

}  // namespace

cudaError_t launch_simrank_walks(const uint32_t* verts, uint32_t nverts, uint32_t R, uint32_t L, gw_walk_rec* out,
                                 cudaStream_t stream) {
  const uint64_t n = (uint64_t)nverts * R;
  if (n == 0) return cudaSuccess;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const uint64_t need = (n + 255) / 256, cap = (uint64_t)sms * 16;
  simrank_walks_kernel<<<(unsigned)(need < cap ? need : cap), 256, 0, stream>>>(verts, n, R, L, out);
  return cudaGetLastError();
}

cudaError_t launch_simrank_meet(const uint32_t* a, const uint32_t* b, const unsigned long long* rows, uint32_t nq,
                                uint32_t R, uint32_t L, unsigned long long* meet, cudaStream_t stream) {
  cudaError_t e = cudaMemsetAsync(meet, 0, (size_t)nq * L * sizeof(unsigned long long), stream);
  if (e != cudaSuccess || R == 0 || L == 0) return e;
  // Comparisons up to which pairs are compared: 12 queries of R = 1000, L = 11
  // take about 38 us so, and about 35 us joined; 64 take 205 and 65.  (1000
  // walks on four vertices, one query: 10 us compared, 370 joined.)
  constexpr uint64_t kPairWork = 1ull << 27;
  const uint64_t compares = (uint64_t)R * R * L;
  const bool join = compares >= kPairWork / std::max(nq, 1u);
  // Joined tiles of 512 walks repeat the hashing least (512 queries: 0.57 ms a
  // call against 0.65 in tiles of 256) but need enough queries to fill the
  // SMs (64 queries: 0.18 against 0.16).
  const uint64_t wide = (R + 511) / 512;
  const uint32_t log = wide * wide * nq >= 592 ? 9 : 8;
  const uint32_t tile = join ? 1u << log : (uint32_t)kPairTile, tiles = (R + tile - 1) / tile;
  const size_t smem = join ? 2 * kSrChunk * (size_t)(tile + 1) * 4 : 0;
  auto k = !join ? simrank_pairs_kernel : log == 9 ? simrank_join_kernel<9> : simrank_join_kernel<8>;
  if (join) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  for (uint32_t q0 = 0; q0 < nq && e == cudaSuccess; q0 += 65535u) {
    const uint32_t nz = nq - q0 < 65535u ? nq - q0 : 65535u;
    k<<<dim3(tiles, tiles, nz), join ? tile : kPairThreads, smem, stream>>>(a, b, rows, q0, R, L, meet);
    e = cudaGetLastError();
  }
  return e;
}

}  // namespace gw
