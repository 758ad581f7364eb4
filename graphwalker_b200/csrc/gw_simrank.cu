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
//    a million per position there), so a CTA marks the vertices of a tile of
//    b's walks in a bitmap and looks a tile of a's walks up in it, O(R) work a
//    position; only a walk whose bit is set is compared with the whole tile,
//    by a warp, two such walks at a time.  A bit per pair in shared memory
//    keeps who has met, as in the pairs kernel, so a matching pair costs one
//    bit, however many match.  111 us for the same queries (251 with the
//    walks in hash chains and each match checked against all earlier
//    positions); bound by issue slots and the latency of two barriers and a
//    few shared-memory round trips per position.  Where walks coincide, most
//    of a tile's are candidates at position after position: tiles of 128 and
//    256 then compare every pair, a thread its walk with all of b's, and look
//    again at every fourth position (one query of 3000 walks x 40 on 16
//    vertices: 241 us a call with candidates alone, 197 all pairs, 185 so; 2000
//    queries of 100 walks x 30 there: 1087, 664, 629).  Tiles of 512 belong to
//    batches that joining serves best even so (512 queries on 16 vertices 977
//    us, 1759 all pairs), and the code would cost them registers.
//
// Every position being a round of such latency, small batches keep comparing
// pairs (kJoinPairs).  The grid's z dimension runs over queries: query q
// compares the R walks at row offset rows[2q] of `a` with those at
// rows[2q + 1] of `b`.
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

constexpr uint32_t kNoVisit = 0xffffffffu;
constexpr uint32_t kSrChunk = 6;  // positions staged at a time (12 leave two CTAs an SM, 4 are read in shorter pieces)

// Every pair of a tile of TILE walks a side at one position: a thread compares
// its walk of a with all of b, and keeps who has met in words (word w of walk i
// at pairs[w * (TILE + 1) + i]) that it alone changes from one such position to
// the next.  Returns the pairs that met now.
template <uint32_t TILE>
__device__ __forceinline__ uint32_t compare_all(const uint32_t* sa, const uint32_t* sb, uint32_t* pairs) {
  const uint32_t p = sa[threadIdx.x];
  uint32_t n = 0;
#pragma unroll 1
  for (uint32_t k = 0; k < TILE / 128; ++k) {
    uint32_t* const mine = pairs + 4 * k * (TILE + 1) + threadIdx.x;
    uint32_t old[4], now[4] = {0, 0, 0, 0};
#pragma unroll
    for (uint32_t e = 0; e < 4; ++e) old[e] = mine[e * (TILE + 1)];
    if (__all_sync(~0u, (old[0] & old[1] & old[2] & old[3]) == ~0u)) continue;
#pragma unroll 8
    for (uint32_t w = 0; w < 32; ++w) {
      const uint4 v = *reinterpret_cast<const uint4*>(sb + 128 * k + 4 * w);
      const uint32_t bit = 1u << w;
      if (p == v.x) now[0] |= bit;
      if (p == v.y) now[1] |= bit;
      if (p == v.z) now[2] |= bit;
      if (p == v.w) now[3] |= bit;
    }
#pragma unroll
    for (uint32_t e = 0; e < 4; ++e) {
      const uint32_t fresh = p == kNoVisit ? 0u : now[e] & ~old[e];
      n += __popc(fresh);
      if (fresh) mine[e * (TILE + 1)] = old[e] | fresh;
    }
  }
  return n;
}

// LOG: a tile is 2^LOG walks of each side, one of each per thread.
template <int LOG>
__global__ void __launch_bounds__(1 << LOG, LOG == 8 ? 8 : 0)
    simrank_join_kernel(const uint32_t* __restrict__ a0, const uint32_t* __restrict__ b0,
                        const unsigned long long* __restrict__ rows, uint32_t q0, uint32_t R, uint32_t L,
                        unsigned long long* __restrict__ meet0) {
  constexpr uint32_t kSrTile = 1 << LOG, kWarps = kSrTile / 32, kRow = kSrTile + 4, kWords = kSrTile / 32;
  constexpr uint32_t kBits = 64 * kSrTile;  // a bit per hashed vertex
  auto bit_of = [](uint32_t v) { return (v * 0x9E3779B1u) >> (26 - LOG); };
  extern __shared__ __align__(16) uint32_t staged[];
  uint32_t(*const sa)[kRow] = reinterpret_cast<uint32_t(*)[kRow]>(staged);
  uint32_t(*const sb)[kRow] = sa + kSrChunk;
  // a bit per pair that has met, word w of walk i of a: by words where threads
  // compare a walk each, by walks where warps do
  uint32_t* const pairs = staged + 2 * kSrChunk * kRow;
  auto pair_word = [&](uint32_t w, uint32_t i) -> uint32_t& {
    return pairs[LOG < 9 ? w * (kSrTile + 1) + i : i * kWords + w];
  };
  __shared__ __align__(16) uint32_t bits[2][kBits / 32];  // one is cleared while the other is read
  __shared__ uint16_t cand[kSrTile];                       // a's walks whose vertex has its bit set
  __shared__ uint32_t ncand[2];
  __shared__ uint32_t found[kSrChunk];  // pairs met at a staged position
  __shared__ uint32_t met;              // pairs of the tile that have met
  const uint32_t q = q0 + blockIdx.z, x = threadIdx.x, lane = x & 31, warp = x >> 5;
  const uint32_t i0 = blockIdx.y * kSrTile, j0 = blockIdx.x * kSrTile;
  const uint32_t na = min(R - i0, kSrTile), nb = min(R - j0, kSrTile);
  const uint32_t* __restrict__ a = a0 + (rows ? rows[2 * (size_t)q] : 0ull) + (size_t)i0 * L;
  const uint32_t* __restrict__ b = b0 + (rows ? rows[2 * (size_t)q + 1] : 0ull) + (size_t)j0 * L;
  unsigned long long* __restrict__ meet = meet0 + (size_t)q * L;
  auto clear = [&](uint32_t t) {
    for (uint32_t w = x; w < kBits / 128; w += kSrTile) reinterpret_cast<uint4*>(bits[t])[w] = make_uint4(0, 0, 0, 0);
  };
  clear(0);
  for (uint32_t w = x; w < kWords * (kSrTile + 1); w += kSrTile) pairs[w] = 0;
  if (x == 0) met = ncand[0] = ncand[1] = 0;
  if (x < kSrChunk) found[x] = 0;
  uint32_t l0 = 0;  // first position staged
  uint32_t t = 0;   // the bitmap in use
  bool dense = false;
  for (uint32_t l = 0; l < L; ++l) {
    const uint32_t c = l % kSrChunk;
    if (LOG == 9) t = l & 1;
    if (c == 0) {
      __syncthreads();  // the candidates before are done with the rows staged before
      if (x < kSrChunk && found[x]) {
        atomicAdd(meet + l0 + x, (unsigned long long)found[x]);
        found[x] = 0;
      }
      const uint32_t w = min(L - l, kSrChunk);  // rows of a tile lie one behind the other
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
    uint32_t count = 0;
    // Where most of a's walks were candidates (all but an eighth in tiles of
    // 256, where a candidate costs less), the next three positions are compared
    // without looking.
    if (!dense || (l & 3u) == 0) {
      // mark b's vertices; half of a position's walks can stand on one vertex
      // (the source they return to), so a bit that is set is left alone
      const uint32_t u = sb[c][x], h = bit_of(u), m = 1u << (h & 31u);
      if (u != kNoVisit && !(*reinterpret_cast<volatile uint32_t*>(&bits[t][h >> 5]) & m)) atomicOr(&bits[t][h >> 5], m);
      __syncthreads();
      if (met == na * nb) break;  // met changes only after the next barrier
      // a's walks that may stand on one of them
      const uint32_t v = sa[c][x], hv = bit_of(v);
      const bool may = v != kNoVisit && ((bits[t][hv >> 5] >> (hv & 31u)) & 1u);
      const uint32_t mine = __ballot_sync(~0u, may);
      if (mine) {
        uint32_t at = 0;
        if (lane == 0) at = atomicAdd(&ncand[t], (uint32_t)__popc(mine));
        at = __shfl_sync(~0u, at, 0) + __popc(mine & ((1u << lane) - 1u));
        if (may) cand[at] = (uint16_t)x;
      }
      clear(t ^ 1);
      if (x == 0) ncand[t ^ 1] = 0;
      __syncthreads();
      count = ncand[t];
      if (LOG < 9) t ^= 1;
      dense = LOG == 7 ? 2 * count > na : LOG == 8 && 8 * count > 7 * na;
    }
    uint32_t n = 0;
    if constexpr (LOG < 9) {
      if (dense) n = compare_all<kSrTile>(sa[c], sb[c], pairs);
    }
    // a warp per two candidates, its lanes over b's walks
    for (uint32_t y = LOG < 9 && dense ? count : 2 * warp; y < count; y += 2 * kWarps) {
      const bool two = y + 1 < count;
      const uint32_t i0 = cand[y], i1 = cand[two ? y + 1 : y], p0 = sa[c][i0], p1 = sa[c][i1];
      uint32_t now0 = 0, now1 = 0;  // lane w: word w of a walk's matches
#pragma unroll
      for (uint32_t k = 0; k < kWords / 4; ++k) {
        const uint4 w = *reinterpret_cast<const uint4*>(&sb[c][4 * lane + 128 * k]);
        auto word = [&](uint32_t p) {
          const uint32_t m0 = __ballot_sync(~0u, w.x == p), m1 = __ballot_sync(~0u, w.y == p);
          const uint32_t m2 = __ballot_sync(~0u, w.z == p), m3 = __ballot_sync(~0u, w.w == p);
          return lane & 2 ? (lane & 1 ? m3 : m2) : (lane & 1 ? m1 : m0);
        };
        const uint32_t w0 = word(p0), w1 = word(p1);
        if (lane / 4 == k) {
          now0 = w0;
          now1 = w1;
        }
      }
      if (now0) {
        const uint32_t old = pair_word(lane, i0);
        n += __popc(now0 & ~old);
        pair_word(lane, i0) = old | now0;
      }
      if (two && now1) {
        const uint32_t old = pair_word(lane, i1);
        n += __popc(now1 & ~old);
        pair_word(lane, i1) = old | now1;
      }
    }
    n = __reduce_add_sync(~0u, n);
    if (lane == 0 && n) {
      atomicAdd(&found[c], n);
      atomicAdd(&met, n);
    }
  }
  __syncthreads();
  if (x < kSrChunk && found[x]) atomicAdd(meet + l0 + x, (unsigned long long)found[x]);
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
  // Pairs of walks from which on they are joined, whatever the length: a
  // position costs a tile the same few round trips, so what counts is how many
  // pairs share them (calls of queries on uniform graphs of 8 edges a vertex, us,
  // compared / joined; 100,000 vertices: one of R = 1000, 50 positions 122 / 136, of
  // 2000 160 / 136, of 3000 214 / 142; 16 of 1000 310 / 158; on 300 vertices 124 / 162,
  // 160 / 172, 222 / 188 and 320 / 235; one of 1000, 135 positions, on 16 vertices 80 /
  // 170).  Up to 64 walks a query, half of the smallest tile joined is empty
  // (5000 queries of 64: 1426 / 1493).
  constexpr uint64_t kJoinPairs = 6000000;
  const bool join = R > 64 && (uint64_t)R * R >= (kJoinPairs + nq - 1) / std::max(nq, 1u);
  // Joined tiles of 512 walks repeat the marking least (a call of 512 queries:
  // 0.30 ms, 0.34 in tiles of 256, 0.44 of 128) but need 592 tiles, four an
  // SM, to fill the chip (24 queries: 107 us, 85 and 93; one dense query of
  // 3000 walks x 40: 717, 379 and 270; all with one walk compared at a time).
  // Queries of up to 256 walks fit no larger one better (1000 of 200 walks, 50
  // positions, 300 vertices: 864 us in tiles of 256, 747 of 128).
  uint32_t log = R > 256 ? 9 : 7;
  for (; log > 7; --log) {
    const uint64_t wide = (R + (1ull << log) - 1) >> log;
    if (wide * wide * nq >= 592) break;
  }
  const uint32_t tile = join ? 1u << log : (uint32_t)kPairTile, tiles = (R + tile - 1) / tile;
  const size_t smem = join ? (2 * kSrChunk * (size_t)(tile + 4) + tile / 32 * (size_t)(tile + 1)) * 4 : 0;
  auto k = !join ? simrank_pairs_kernel
           : log == 9 ? simrank_join_kernel<9> : log == 8 ? simrank_join_kernel<8> : simrank_join_kernel<7>;
  if (join) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  for (uint32_t q0 = 0; q0 < nq && e == cudaSuccess; q0 += 65535u) {
    const uint32_t nz = nq - q0 < 65535u ? nq - q0 : 65535u;
    k<<<dim3(tiles, tiles, nz), join ? tile : kPairThreads, smem, stream>>>(a, b, rows, q0, R, L, meet);
    e = cudaGetLastError();
  }
  return e;
}

}  // namespace gw
