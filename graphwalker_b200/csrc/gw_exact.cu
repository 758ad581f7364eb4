// gw_exact.cu -- expected visits per vertex of one walk from a source, in
// FP64, by propagating the exact per-hop distribution over the resident
// graph (the truncated power series behind PPR / RWR estimates).
//
// x_0 = e_src.  Each hop: a vertex with out-edges passes x[v]*q/deg to every
// out-neighbour (q = the exact probability that a 31-bit draw passes the
// continuation test); the rest -- x[v]*(1-q), or all of x[v] at a dangling
// vertex -- follows the rule's else-branch: back to the source (restart; the
// PPR rule only at dangling vertices), spread uniformly (jump), or ends (stop).
// Visits accumulate x_h for every hop the rule visits (L hops for the capped
// rules, L-1 per restart segment, until the mass vanishes for the uncapped
// rule).  The neighbour choice is taken as exactly uniform; the walks'
// r % deg has a bias below deg / 2^31.
//
// A hop is two kernels.  The vertex kernel finishes x (what arrived over edges
// plus what the last hop's else-branches owe the source and all vertices), adds
// it to the visits, leaves each vertex's share per out-edge and sums the new
// debts.  The edge kernel carries the shares to the targets, warps taking equal
// runs of edges whatever their vertices' degrees, so no warp is left with a
// hub: a warp per vertex took 355 us a hop at R-MAT scale 20 (16.8 M edges).
//
//  * Push: an FP64 atomic per edge, 154 us a hop there, the L2's rate of them
//    (109 G/s; 32-bit ones: 190).  It is not the hottest target's address:
//    pushes spread over 2 or 4 copies of the targets gained 5 % and lost 11 %.
//  * Pull: over in-edges, so an edge is a gather (284 G/s from the L2) and only
//    the end of a vertex's run of edges an atomic: 85 us a hop, after 385 us of
//    turning the graph around, a counting sort by target.  The first pushes
//    cost little, as few vertices have been reached: pull_from says from how
//    many hops on a call pulls.
#include <algorithm>

#include "gw_ctx.h"

namespace gw {
namespace {

constexpr int kExactThreads = 256;
constexpr int kSums = 4;  // debt sets: the last hop's, this one's, and one cleared ahead

struct Debt {
  double to_src, to_uniform, mass;
};

__device__ __forceinline__ double block_sum(double v, double* warp_sums) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(~0u, v, o);
  if ((threadIdx.x & 31) == 0) warp_sums[threadIdx.x >> 5] = v;
  __syncthreads();
  v = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < kExactThreads / 32; ++w) v += warp_sums[w];
  __syncthreads();
  return v;  // in thread 0
}

// x (in acc) of this hop; acc is left zero for the edge kernel's pushes.
__global__ void __launch_bounds__(kExactThreads)
    exact_vertex_kernel(double* __restrict__ acc, double* __restrict__ share, double* __restrict__ visits,
                        Debt* __restrict__ debts, uint32_t hop, const unsigned long long* __restrict__ rowptr,
                        uint32_t nv, uint32_t src, uint32_t njump, double q, int rule) {
  __shared__ double warp_sums[kExactThreads / 32];
  const Debt last = debts[(hop + kSums - 1) % kSums];  // zero before the first hop
  if (blockIdx.x == 0 && threadIdx.x == 0) debts[(hop + 1) % kSums] = Debt{0.0, 0.0, 0.0};
  const double uniform = last.to_uniform / (double)njump;
  double to_src = 0.0, to_uniform = 0.0, mass = 0.0;
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += (uint64_t)gridDim.x * blockDim.x) {
    double add = v < njump ? uniform : 0.0;
    if (v == src) add += last.to_src;
    const double xv = acc[v] + add;
    double sh = 0.0;
    if (xv != 0.0) {
      const unsigned long long deg = rowptr[v + 1] - rowptr[v];
      visits[v] += xv;
      mass += xv;
      double fail = xv;
      if (deg > 0) {
        sh = xv * q / (double)deg;
        fail = xv * (1.0 - q);
      }
      if (rule == GW_RULE_RESTART || (rule == GW_RULE_PPR && deg == 0)) to_src += fail;
      else if (rule == GW_RULE_JUMP) to_uniform += fail;
    }
    share[v] = sh;
    acc[v] = 0.0;
  }
  to_src = block_sum(to_src, warp_sums);
  to_uniform = block_sum(to_uniform, warp_sums);
  mass = block_sum(mass, warp_sums);
  if (threadIdx.x == 0) {
    Debt* d = debts + hop % kSums;
    if (to_src != 0.0) atomicAdd(&d->to_src, to_src);
    if (to_uniform != 0.0) atomicAdd(&d->to_uniform, to_uniform);
    if (mass != 0.0) atomicAdd(&d->mass, mass);
  }
}

// first[c]: the source of edge c * run (the last vertex whose row starts at or
// before it and is not empty).
__global__ void exact_runs_kernel(const unsigned long long* __restrict__ rowptr, uint32_t nv, uint64_t nruns,
                                  uint32_t run, uint32_t* __restrict__ first) {
  for (uint64_t c = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; c < nruns; c += (uint64_t)gridDim.x * blockDim.x) {
    const unsigned long long e = c * run;
    uint32_t lo = 0, hi = nv;  // first v with rowptr[v + 1] > e
    while (lo < hi) {
      const uint32_t mid = lo + (hi - lo) / 2;
      if (rowptr[mid + 1] > e) hi = mid;
      else lo = mid + 1;
    }
    first[c] = lo;
  }
}

// The lane whose row holds edge e, when lane i's row ends at `end` (in lane
// order) and e lies in one of them: the number of rows that end at or before e.
__device__ __forceinline__ uint32_t row_of(uint32_t end, uint32_t e) {
  uint32_t at = 0;
#pragma unroll
  for (uint32_t step = 16; step > 0; step >>= 1)
    if (__shfl_sync(~0u, end, at + step - 1) <= e) at += step;
  return at;
}

// The first group of 32 rows, a multiple of 32 past v, that holds an edge past
// e, or nv: a warp looks at the ends of 32 groups at a time, then of 32 times
// as many, so a stretch of rows without edges costs its logarithm and not a
// load for every 32 of them.  A call over a million vertices with 150 edges at
// either end: three pushes 29.8 ms row group by row group, 1.3 so; nine pulls
// 86.7 and 1.5.  Not inlined: runs that never need it pay for its code (scale
// 16, 20 hops: 488 us a call, 527 with it inline).
__device__ __noinline__ uint32_t next_rows(const unsigned long long* __restrict__ rows, uint32_t nv,
                                           unsigned long long e, uint32_t v, uint32_t lane) {
  uint32_t width = 32;  // rows a lane stands for
  while (v < nv) {
    const uint64_t row = (uint64_t)v + (uint64_t)(lane + 1) * width - 1;
    const uint32_t ends = __ballot_sync(~0u, __ldg(rows + (row < nv ? row : nv - 1) + 1) > e);
    if (ends) {  // inside the first such lane's rows
      v += (uint32_t)(__ffs(ends) - 1) * width;
      if (width == 32) return v;
      width /= 32;
    } else {
      if ((uint64_t)v + 32ull * width >= nv) break;
      v += 32 * width;
      if (width < 1u << 20) width *= 32;
    }
  }
  return nv;
}

// One warp per run of edges of the rows `rowptr`, which are sources; the lanes
// hold the row ends of 32 consecutive ones.  Push: a row's share is added at
// each of its targets.  Turn: a row's source is written into each target's row
// of the turned graph, whose next free place is place[target].  An edge to a
// vertex past the last carries nothing.
template <bool TURN>
__global__ void __launch_bounds__(kExactThreads)
    exact_edge_kernel(const double* __restrict__ share, double* __restrict__ acc,
                      const unsigned long long* __restrict__ rowptr, const uint32_t* __restrict__ colidx, uint32_t nv,
                      uint64_t ne, uint64_t nruns, uint32_t run, const uint32_t* __restrict__ first,
                      uint32_t* __restrict__ place, uint32_t* __restrict__ turned) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t c = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (c >= nruns) return;
  const uint64_t e0 = c * run;
  const uint32_t n = (uint32_t)(ne - e0 < run ? ne - e0 : run);  // positions below are relative to e0
  uint32_t v = __ldg(first + c);
  for (uint32_t done = 0; done < n; v += 32) {
    const uint32_t mine = v + lane;
    uint32_t end = n;  // of vertex `mine`, at most n
    double sh = 0.0;
    if (mine < nv) {
      const unsigned long long x = __ldg(rowptr + mine + 1) - e0;
      end = x < n ? (uint32_t)x : n;
      if (!TURN) sh = __ldg(share + mine);
    }
    const uint32_t last = __shfl_sync(~0u, end, 31);  // edges these vertices reach to
    if (__builtin_expect(last == done, 0)) {
      v = next_rows(rowptr, nv, e0 + done, v + 32, lane) - 32;
      continue;
    }
    const bool any = TURN || __any_sync(~0u, sh != 0.0);
    for (; any && done < last; done += 128) {
      uint32_t to[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint32_t e = done + u * 32 + lane;
        to[u] = e < last ? __ldg(colidx + e0 + e) : nv;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint32_t at = row_of(end, done + u * 32 + lane);
        const double s = TURN ? 0.0 : __shfl_sync(~0u, sh, at);
        if (to[u] >= nv) continue;
        if (TURN) turned[atomicAdd(place + to[u], 1u)] = v + at;
        else if (s != 0.0) atomicAdd(acc + to[u], s);
      }
    }
    done = last;
  }
}

// The same over the turned graph: rows are targets, turned[e] the source of
// in-edge e.  A lane sums four consecutive edges; where they span rows it adds
// all but the last row's part by itself, and the last parts of the lanes of one
// row are summed in the warp and added by its first lane.
__global__ void __launch_bounds__(kExactThreads)
    exact_pull_kernel(const double* __restrict__ share, double* __restrict__ acc,
                      const unsigned long long* __restrict__ rows, const uint32_t* __restrict__ turned, uint32_t nv,
                      uint64_t ne, uint64_t nruns, uint32_t run, const uint32_t* __restrict__ first) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t c = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (c >= nruns) return;
  const uint64_t e0 = c * run;
  const uint32_t n = (uint32_t)(ne - e0 < run ? ne - e0 : run);
  uint32_t v = __ldg(first + c);
  for (uint32_t done = 0; done < n && v < nv; v += 32) {
    const uint32_t mine = v + lane;
    uint32_t end = n;
    if (mine < nv) {
      const unsigned long long x = __ldg(rows + mine + 1) - e0;
      end = x < n ? (uint32_t)x : n;
    }
    const uint32_t last = __shfl_sync(~0u, end, 31);
    if (__builtin_expect(last == done, 0)) {
      v = next_rows(rows, nv, e0 + done, v + 32, lane) - 32;
      continue;
    }
    for (; done < last; done += 128) {
      const uint32_t e = done + lane * 4;
      uint32_t src[4], at[4];
      double got[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) src[u] = e + u < last ? __ldg(turned + e0 + e + u) : nv;
#pragma unroll
      for (int u = 0; u < 4; ++u) got[u] = src[u] < nv ? __ldg(share + src[u]) : 0.0;
#pragma unroll
      for (int u = 0; u < 4; ++u) at[u] = row_of(end, e + u);
      double s = got[0];
#pragma unroll
      for (int u = 1; u < 4; ++u) {
        if (at[u] != at[u - 1]) {
          if (s != 0.0 && v + at[u - 1] < nv) atomicAdd(acc + v + at[u - 1], s);
          s = 0.0;
        }
        s += got[u];
      }
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double x = __shfl_down_sync(~0u, s, o);
        const uint32_t row = __shfl_down_sync(~0u, at[3], o);
        if (lane + o < 32 && row == at[3]) s += x;
      }
      const uint32_t before = __shfl_up_sync(~0u, at[3], 1);
      if ((lane == 0 || before != at[3]) && s != 0.0 && v + at[3] < nv) atomicAdd(acc + v + at[3], s);
    }
    done = last;
  }
}

// In-degrees of the turned graph.
__global__ void in_degree_kernel(const uint32_t* __restrict__ colidx, uint64_t ne, uint32_t nv,
                                 uint32_t* __restrict__ deg) {
  for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < ne; e += (uint64_t)gridDim.x * blockDim.x)
    if (const uint32_t to = __ldg(colidx + e); to < nv) atomicAdd(deg + to, 1u);
}

// Exclusive scan of the in-degrees, in three launches: every block's sum; the
// sums, in one block; then rows[v] (where v's in-edges start) and place[v] (the
// same, advanced by the turn; it holds the in-degrees before).
constexpr uint32_t kScanItems = 4, kScanBlock = kExactThreads * kScanItems;

__device__ __forceinline__ unsigned long long block_scan(unsigned long long x, unsigned long long* warp_sums,
                                                         unsigned long long* total) {
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long incl = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long y = __shfl_up_sync(~0u, incl, o);
    if (lane >= (uint32_t)o) incl += y;
  }
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  unsigned long long below = 0, all = 0;
  for (uint32_t w = 0; w < kExactThreads / 32; ++w) {
    if (w < warp) below += warp_sums[w];
    all += warp_sums[w];
  }
  __syncthreads();  // warp_sums may be written again
  *total = all;
  return below + incl - x;
}

__global__ void __launch_bounds__(kExactThreads)
    scan_sums_kernel(const uint32_t* __restrict__ deg, uint32_t nv, unsigned long long* __restrict__ sums) {
  __shared__ unsigned long long warp_sums[kExactThreads / 32];
  const uint64_t v0 = (uint64_t)blockIdx.x * kScanBlock + threadIdx.x * kScanItems;
  unsigned long long x = 0, all = 0;
  for (uint32_t i = 0; i < kScanItems; ++i)
    if (v0 + i < nv) x += deg[v0 + i];
  block_scan(x, warp_sums, &all);
  if (threadIdx.x == 0) sums[blockIdx.x] = all;
}

__global__ void __launch_bounds__(kExactThreads) scan_blocks_kernel(unsigned long long* __restrict__ sums, uint32_t n) {
  __shared__ unsigned long long warp_sums[kExactThreads / 32];
  unsigned long long carry = 0;
  for (uint32_t b = 0; b < n; b += kExactThreads) {
    const uint32_t i = b + threadIdx.x;
    const unsigned long long x = i < n ? sums[i] : 0ull;
    unsigned long long all = 0;
    const unsigned long long before = block_scan(x, warp_sums, &all);
    if (i < n) sums[i] = carry + before;
    carry += all;
  }
}

__global__ void __launch_bounds__(kExactThreads)
    scan_rows_kernel(uint32_t* __restrict__ place, uint32_t nv, const unsigned long long* __restrict__ sums,
                     unsigned long long* __restrict__ rows) {
  __shared__ unsigned long long warp_sums[kExactThreads / 32];
  const uint64_t v0 = (uint64_t)blockIdx.x * kScanBlock + threadIdx.x * kScanItems;
  uint32_t d[kScanItems];
  unsigned long long x = 0, all = 0;
#pragma unroll
  for (uint32_t i = 0; i < kScanItems; ++i) {
    d[i] = v0 + i < nv ? place[v0 + i] : 0u;
    x += d[i];
  }
  unsigned long long at = sums[blockIdx.x] + block_scan(x, warp_sums, &all);
#pragma unroll
  for (uint32_t i = 0; i < kScanItems; ++i) {
    if (v0 + i >= nv) break;
    rows[v0 + i] = at;
    place[v0 + i] = (uint32_t)at;
    at += d[i];
    if (v0 + i + 1 == nv) rows[nv] = at;
  }
}

// The workspace is kept in the context up to this size.
constexpr size_t kKeptBytes = 256ull << 20;

// The hops from which a call pulls instead of pushing, with a workspace of
// `bytes` then.  Turning the graph around costs what 4 to 8 pulls do; a push of
// a graph of average degree 16 costs about two pulls once all vertices are
// reached, which takes a few hops, and fewer with a higher degree (calls from
// the vertex of highest degree, pushed / pulled, us: scale 16, 8 hops 341 / 315;
// scale 18, 8 hops 788 / 786, 10 hops 922 / 856; scale 20, 8 hops 2127 / 2263,
// 12 hops 2742 / 2670; scale 19 and degree 48, 8 hops 2122 / 2088; from a vertex
// of degree 1 pulling pays two hops later).  Below 2^17 edges a call is a chain
// of launches, and the turn's are six more (scale 12, 20 hops: 258 / 294; the
// uncapped rule, some hundred: 2588 / 2336).  A workspace too large to keep is allocated by each call, and the turn's
// scattered writes leave the L2 (scale 24, from a vertex of degree 1, 7 hops: 58 ms
// with a warp per vertex pushing, 71 pulled; 20 hops from the highest: 113 / 103).
uint32_t pull_from(uint64_t nv, uint64_t ne, size_t bytes) {
  if (ne == 0 || ne >= 1ull << 32) return 0xffffffffu;  // never (places are 32 bits)
  if (ne < 1ull << 17) return 48;
  if (bytes > kKeptBytes) return 20;
  return ne < 1ull << 22 || ne >= 32 * nv ? 8 : 12;
}

}  // namespace
}  // namespace gw

extern "C" gw_status gw_expected_visits(gw_ctx* ctx, const gw_walk_params* params, uint32_t source, double* out) {
  if (!ctx) return GW_E_INVALID;
  if (ctx->residency != GW_RESIDENT_HBM) return ctx->fail(GW_E_STATE, "needs a resident graph");
  if (!out || source >= ctx->nv) return ctx->fail(GW_E_INVALID, "bad source or NULL output");
  gw::WalkArgs a;
  gw_status s = gw::make_walk_args(ctx, params, &a);
  if (s != GW_OK) return s;
  const double q = (double)(0x80000000u - a.thr) / 2147483648.0;
  const int rule = (int)params->rule;
  uint32_t hops;
  if (rule == GW_RULE_RESTART) hops = params->L > 1 ? params->L - 1 : 1;
  else if (rule == GW_RULE_PROB) hops = a.max_hops;
  else hops = params->L;
  const size_t nv = ctx->nv;
  GW_CUDA(ctx, cudaSetDevice(ctx->device), "cudaSetDevice");
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
  // Edges per warp: enough warps to fill the SMs, at most 1024 edges each.
  const uint64_t ne = ctx->ne;
  const uint32_t run = (uint32_t)std::min<uint64_t>(std::max<uint64_t>(ne / ((uint64_t)sms * 64) / 128 * 128, 128), 1024);
  const uint64_t nruns = (ne + run - 1) / run;
  // One workspace: arrivals, shares and visits (8 bytes a vertex each), the debt
  // sets, the turned graph's rows (8 bytes a vertex) and block sums, the runs'
  // first vertices, and the turned graph's places (4 bytes a vertex) and sources
  // (4 bytes an edge).
  bool pull = true;
  const uint32_t nscan = (uint32_t)((nv + gw::kScanBlock - 1) / gw::kScanBlock);
  const size_t debts_at = 3 * nv * 8, rows_at = debts_at + gw::kSums * sizeof(gw::Debt);
  size_t first_at = 0, place_at = 0, turned_at = 0;
  auto lay_out = [&] {
    first_at = rows_at + (pull ? (nv + 1 + nscan) * 8 : 0);
    place_at = first_at + nruns * 4;
    turned_at = place_at + (pull ? nv * 4 : 0);
    return turned_at + (pull ? ne * 4 : 0);
  };
  pull = hops >= gw::pull_from(nv, ne, lay_out());
  if (pull && ctx->d_exact.ensure(lay_out()) != cudaSuccess) {
    cudaGetLastError();  // no room to turn the graph around: push
    pull = false;
  }
  GW_CUDA(ctx, ctx->d_exact.ensure(lay_out()), "alloc");
  struct Release {
    gw_ctx* ctx;
    ~Release() {
      if (ctx->d_exact.bytes > gw::kKeptBytes) ctx->d_exact.release();
    }
  } release{ctx};
  cudaStream_t st = ctx->stream;
  double* acc = ctx->d_exact.as<double>();
  double *share = acc + nv, *visits = share + nv;
  gw::Debt* debts = reinterpret_cast<gw::Debt*>(ctx->d_exact.as<char>() + debts_at);
  uint32_t* first = reinterpret_cast<uint32_t*>(ctx->d_exact.as<char>() + first_at);
  GW_CUDA(ctx, cudaMemsetAsync(acc, 0, nv * 8, st), "clear");
  GW_CUDA(ctx, cudaMemsetAsync(visits, 0, nv * 8 + gw::kSums * sizeof(gw::Debt), st), "clear");  // and the debts
  const double one = 1.0;
  GW_CUDA(ctx, cudaMemcpyAsync(acc + source, &one, 8, cudaMemcpyHostToDevice, st), "seed");
  const unsigned long long* rowptr = ctx->d_rowptr.as<unsigned long long>();
  const uint32_t* const colidx = ctx->d_colidx.as<uint32_t>();
  const unsigned egrid = (unsigned)((nruns * 32 + gw::kExactThreads - 1) / gw::kExactThreads);
  const unsigned rgrid = (unsigned)std::min<uint64_t>((nruns + 255) / 256, (uint64_t)sms * 8);
  auto* rows = reinterpret_cast<unsigned long long*>(ctx->d_exact.as<char>() + rows_at);
  uint32_t* const turned = reinterpret_cast<uint32_t*>(ctx->d_exact.as<char>() + turned_at);
  if (nruns) {
    gw::exact_runs_kernel<<<rgrid, 256, 0, st>>>(rowptr, ctx->nv, nruns, run, first);
    GW_CUDA(ctx, cudaGetLastError(), "edge runs");
  }
  if (pull) {
    unsigned long long* const sums = rows + nv + 1;
    uint32_t* const place = reinterpret_cast<uint32_t*>(ctx->d_exact.as<char>() + place_at);
    GW_CUDA(ctx, cudaMemsetAsync(place, 0, nv * 4, st), "clear");
    gw::in_degree_kernel<<<(unsigned)std::min<uint64_t>((ne + 255) / 256, (uint64_t)sms * 8), 256, 0, st>>>(
        colidx, ne, ctx->nv, place);
    gw::scan_sums_kernel<<<nscan, gw::kExactThreads, 0, st>>>(place, ctx->nv, sums);
    gw::scan_blocks_kernel<<<1, gw::kExactThreads, 0, st>>>(sums, nscan);
    gw::scan_rows_kernel<<<nscan, gw::kExactThreads, 0, st>>>(place, ctx->nv, sums, rows);
    gw::exact_edge_kernel<true><<<egrid, gw::kExactThreads, 0, st>>>(nullptr, nullptr, rowptr, colidx, ctx->nv, ne,
                                                                         nruns, run, first, place, turned);
    gw::exact_runs_kernel<<<rgrid, 256, 0, st>>>(rows, ctx->nv, nruns, run, first);
    GW_CUDA(ctx, cudaGetLastError(), "turn");
  }
  const unsigned vgrid = (unsigned)std::min<uint64_t>((nv + gw::kExactThreads - 1) / gw::kExactThreads, (uint64_t)sms * 8);
  for (uint32_t h = 0; h < hops; ++h) {
    gw::exact_vertex_kernel<<<vgrid, gw::kExactThreads, 0, st>>>(acc, share, visits, debts, h, rowptr, ctx->nv, source,
                                                                 a.njump, q, rule);
    GW_CUDA(ctx, cudaGetLastError(), "exact vertices");
    if (h + 1 == hops) break;  // the last hop's moves are not visited
    if (nruns) {
      if (pull)
        gw::exact_pull_kernel<<<egrid, gw::kExactThreads, 0, st>>>(share, acc, rows, turned, ctx->nv, ne, nruns, run,
                                                                  first);
      else
        gw::exact_edge_kernel<false><<<egrid, gw::kExactThreads, 0, st>>>(share, acc, rowptr, colidx, ctx->nv, ne,
                                                                             nruns, run, first, nullptr, nullptr);
      GW_CUDA(ctx, cudaGetLastError(), "exact edges");
    }
    if (rule == GW_RULE_PROB && (h & 15) == 15) {  // the uncapped rule stops when the mass is gone
      double mass = 0.0;
      GW_CUDA(ctx, cudaMemcpyAsync(&mass, &debts[h % gw::kSums].mass, 8, cudaMemcpyDeviceToHost, st), "mass");
      GW_CUDA(ctx, cudaStreamSynchronize(st), "sync");
      if (mass < 1e-16) break;
    }
  }
  GW_CUDA(ctx, cudaMemcpyAsync(out, visits, nv * 8, cudaMemcpyDeviceToHost, st), "visits out");
  GW_CUDA(ctx, cudaStreamSynchronize(st), "sync");
  return GW_OK;
}
