// brt_order.cu -- the step's order on (cell, agent id) by counting the cells.
//
// The result is the same permutation the stable radix sort of (key, slot)
// pairs in agent-id order produces (RadixSort, radixsort.cu:50-80: keys
// ascending, ties by agent id), from nothing but the current state:
//   countKernel   every agent's cell, and its place among the agents that
//                 reached that cell's counter (in whatever order they came);
//   cellScanKernel  exclusive scan of the counts (single pass, warp-wide
//                 decoupled look-back, bounded waits): the cells' ranges.
//                 It leaves the counts at zero for the next step;
//   placeKernel   every agent to its cell's range, at its place;
//   reorderKernel<true> (brt_kernels.cu)  every agent's rank by id among its
//                 cell's members, and with it the sorted position its state
//                 is copied to.
// A cell holds a few agents, so ranking them by comparing ids is cheaper than
// sorting: four launches take the place of the histogram, the radix passes and
// the reorder.  In a crowded cell (more than kRankLimit agents) comparing all pairs
// would not be: placeKernel sorts those by id.
//
// The kernels are bound by latency (small worlds) or by their scattered 4 to 16
// byte accesses (large ones).  Measured, us of a warm step for all launches
// before the flock kernel, against repairing the previous order (mark, cell scan,
// place, with the hash and radix launches there but gated off): 4,096 agents 13.0
// against 29; 100,003: 17.7 against 38; 1,048,576 with 8 features: 65 against 87;
// 1,024 flocks, 10.2 M agents: 385 against 550.  After a changed state, where the
// radix sort ran: 13 against 30 (4,096), 65 against 108 (1,048,576).  Crowded worlds:
// kRankLimit; worlds of few cells take the radix sort (ordersByCount).
#include "brt_kernels.cuh"

#include <algorithm>

namespace brt {
namespace {

// Cell-scan tiles: THREADS threads of ITEMS consecutive cells, chosen per grid
// (cellScanTile) for about kCellScanTilesTarget tiles: enough to fill the
// GPU, few enough that the look-back stays short when every tile reaches it
// at once.  Small grids take 256-thread tiles of 1 to 4 cells a thread, large
// ones 1024-thread tiles of 8.
constexpr uint32_t kCellScanTilesTarget = 4 * 148;
constexpr uint32_t kLookAgg = 1u << 30;
constexpr uint32_t kLookInc = 2u << 30;
constexpr uint32_t kLookMask = 3u << 30;
constexpr uint32_t kLookVal = (1u << 30) - 1u;
constexpr uint32_t kPlaceThreads = 256;

// Exclusive scan of one value per thread across the CTA (THREADS a multiple
// of 32, at most 1024); the CTA total goes to *total.
template <uint32_t THREADS>
__device__ __forceinline__ uint32_t ctaExclusiveScan(uint32_t v, uint32_t* sWarp, uint32_t* total) {
  constexpr uint32_t WARPS = THREADS / 32;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= (uint32_t)o) x += y;
  }
  if (lane == 31) sWarp[warp] = x;
  __syncthreads();
  if (warp == 0) {
    const uint32_t w = lane < WARPS ? sWarp[lane] : 0u;
    uint32_t wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= (uint32_t)o) wi += y;
    }
    if (lane < WARPS) sWarp[lane] = wi - w;
    if (lane == WARPS - 1) sWarp[WARPS] = wi;
  }
  __syncthreads();
  const uint32_t r = sWarp[warp] + x - v;
  *total = sWarp[WARPS];
  __syncthreads();
  return r;
}

// Agents are in the previous step's order, so neighbouring lanes mostly share
// a cell: one atomic a run of equal cells (its first lane adds the run's
// length), about a quarter of one an agent at 4 agents a cell.
template <bool CHAIN>
__global__ void __launch_bounds__(256) countKernel(OrderArgs A, uint32_t cellTiles) {
  chainBegin();
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < cellTiles) A.tileStatus[j] = 0u;
  if (j == 0) {
    A.words[kOrderWordTile] = 0u;
    A.words[kOrderWordDone] = 0u;
    A.words[kOrderWordBig] = 0u;
    A.words[kOrderWordGiant] = 0u;
    A.words[kOrderWordItem] = 0u;
    if (A.stepCounter) *A.stepCounter += 1u;
  }
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t key = 0xFFFFFFFFu;
  if (j < A.n) {
    const float4 p = ldStep<CHAIN>(&A.pos[j]);
    const FlockDev& fl = A.flocks[A.nflocks == 1 ? 0u : flockOfSlotInWarp(A.agentBase, A.nflocks, j)];
    const int gx = gridCoord(p.x, fl), gy = gridCoord(p.y, fl), gz = gridCoord(p.z, fl);
    key = fl.cellBase + ((uint32_t)gz * fl.G + (uint32_t)gy) * fl.G + (uint32_t)gx;
  }
  const uint32_t before = __shfl_up_sync(0xFFFFFFFFu, key, 1);
  const bool head = lane == 0 || before != key;
  const uint32_t heads = __ballot_sync(0xFFFFFFFFu, head);
  const uint32_t at = 31u - (uint32_t)__clz((int)(heads & (0xFFFFFFFFu >> (31u - lane))));  // this run's first lane
  const uint32_t after = heads & ~(0xFFFFFFFFu >> (31u - lane));
  const uint32_t end = after ? (uint32_t)__ffs((int)after) - 1u : 32u;
  uint32_t first = 0;
  if (head && j < A.n) first = atomicAdd(&A.count[key], end - lane);
  first = __shfl_sync(0xFFFFFFFFu, first, at);
  if (j < A.n) A.cellPlace[j] = make_uint2(key, first + lane - at);
}

template <uint32_t THREADS, uint32_t ITEMS>
__global__ void __launch_bounds__(THREADS) cellScanKernel(OrderArgs A) {
  __shared__ uint32_t sTile, sPrefix;
  __shared__ uint32_t sWarp[THREADS / 32 + 1];
  chainBegin();
  if (threadIdx.x == 0) sTile = atomicAdd(&A.words[kOrderWordTile], 1u);
  __syncthreads();
  const uint32_t tile = sTile;
  const uint32_t c0 = tile * THREADS * ITEMS + threadIdx.x * ITEMS;
  uint32_t tot[ITEMS];
  uint32_t sum = 0;
  // the arrays are padded to whole 16-byte pieces (and beyond the last cell
  // the counts stay zero)
  if constexpr (ITEMS % 4 == 0) {
#pragma unroll
    for (uint32_t k = 0; k < ITEMS; k += 4) {
      const uint4 v = c0 + k < A.numCells ? *reinterpret_cast<const uint4*>(A.count + c0 + k) : make_uint4(0u, 0u, 0u, 0u);
      tot[k] = v.x; tot[k + 1] = v.y; tot[k + 2] = v.z; tot[k + 3] = v.w;
    }
  } else {
#pragma unroll
    for (uint32_t k = 0; k < ITEMS; ++k) tot[k] = c0 + k < A.numCells ? A.count[c0 + k] : 0u;
  }
#pragma unroll
  for (uint32_t k = 0; k < ITEMS; ++k) sum += tot[k];
  uint32_t tileTotal;
  const uint32_t excl = ctaExclusiveScan<THREADS>(sum, sWarp, &tileTotal);
  if (threadIdx.x < 32) {
    // Warp-wide look-back: lane k reads predecessor p - k, so one round
    // covers 32 tiles (tiles that start together would otherwise walk back
    // one dependent load per predecessor).
    const uint32_t lane = threadIdx.x;
    uint32_t before = 0;
    if (tile == 0) {
      if (lane == 0) stRelaxed(&A.tileStatus[0], kLookInc | (tileTotal & kLookVal));
    } else {
      if (lane == 0) stRelaxed(&A.tileStatus[tile], kLookAgg | (tileTotal & kLookVal));
      int p = (int)tile - 1;
      uint32_t spins = 0;
      const bool stalled = tile == A.wait.stallTile;
      while (p >= 0) {
        const int q = p - (int)lane;
        // before tile 0 there is nothing: read as an inclusive zero
        const uint32_t v = q >= 0 ? (stalled ? 0u : ldRelaxed(&A.tileStatus[q])) : kLookInc;
        const uint32_t f = v & kLookMask;
        const uint32_t inc = __ballot_sync(0xffffffffu, f == kLookInc);
        const uint32_t unpublished = __ballot_sync(0xffffffffu, f == 0u);
        const uint32_t first = inc ? (uint32_t)__ffs(inc) - 1u : 31u;  // nearest inclusive prefix
        const uint32_t need = first == 31u ? 0xffffffffu : ((2u << first) - 1u);
        if (unpublished & need) {
          // a predecessor that claimed its tile is resident and publishes soon
          if (++spins > A.wait.spinLimit) {
            if (lane == 0) atomicOr(A.errWord, kDevErrLookback);
            break;
          }
          continue;
        }
        uint32_t add = lane <= first ? (v & kLookVal) : 0u;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) add += __shfl_xor_sync(0xffffffffu, add, o);
        before += add;
        if (inc) break;
        p -= 32;
      }
      if (lane == 0) stRelaxed(&A.tileStatus[tile], kLookInc | ((before + tileTotal) & kLookVal));
    }
    if (lane == 0) sPrefix = before;
  }
  __syncthreads();
  uint32_t run = sPrefix + excl;
  uint32_t start[ITEMS], stop[ITEMS];
#pragma unroll
  for (uint32_t k = 0; k < ITEMS; ++k) {
    start[k] = tot[k] ? run : kEmpty;
    run += tot[k];
    stop[k] = tot[k] ? run : kEmpty;
    if (tot[k] > kRankLimit) {
      const bool giant = tot[k] > giantLimit(A.n);
      const uint32_t b = atomicAdd(&A.words[giant ? kOrderWordGiant : kOrderWordBig], 1u);
      if (giant && b < kGiants) A.giantCells[b] = c0 + k;
      if (!giant && b < bigCellCap(A.n)) A.bigCells[b] = c0 + k;
    }
  }
  if constexpr (ITEMS % 4 == 0) {
#pragma unroll
    for (uint32_t k = 0; k < ITEMS; k += 4) {
      if (c0 + k < A.numCells) {
        *reinterpret_cast<uint4*>(A.cellStart + c0 + k) = make_uint4(start[k], start[k + 1], start[k + 2], start[k + 3]);
        *reinterpret_cast<uint4*>(A.cellEnd + c0 + k) = make_uint4(stop[k], stop[k + 1], stop[k + 2], stop[k + 3]);
        *reinterpret_cast<uint4*>(A.count + c0 + k) = make_uint4(0u, 0u, 0u, 0u);
      }
    }
  } else {
#pragma unroll
    for (uint32_t k = 0; k < ITEMS; ++k) {
      if (c0 + k < A.numCells) {
        A.cellStart[c0 + k] = start[k];
        A.cellEnd[c0 + k] = stop[k];
        A.count[c0 + k] = 0u;
      }
    }
  }
}

// What a block needs while it sorts crowded cells.
struct CrowdShared {
  uint32_t base[kGiants], start[kGiants], end[kGiants], cell[kGiants];
  uint16_t count[kPlaceThreads / 32][256];
  uint32_t warp[kPlaceThreads / 32 + 1];
  uint32_t item;
};
static_assert(kPlaceThreads == 256 && kGiants == 256, "a thread per digit and per giant cell");

// One crowded cell's members, sorted by id: a stable radix sort on 8-bit
// digits by one CTA of kPlaceThreads threads, 256 members at a time, between
// members (id, slot), a pair buffer and the places, which nobody reads any more.
__device__ void sortBigCell(const OrderArgs& A, CrowdShared& S, uint32_t s, uint32_t e, uint32_t key) {
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  uint2* const buf[2] = {A.cellPlace, A.scratch[1]};
  for (uint32_t i = s + tid; i < e; i += kPlaceThreads) {
    const uint4 m = __ldcg(&A.members[i]);
    buf[0][i] = make_uint2(m.x, m.y);
  }
  uint32_t from = 0;
  for (uint32_t shift = 0; shift < 32u && (A.n - 1u) >> shift; shift += 8u, from ^= 1u) {
    const uint2* in = buf[from];
    uint2* out = buf[from ^ 1u];
    S.base[tid] = 0u;
    __syncthreads();
    for (uint32_t i = s + tid; i < e; i += kPlaceThreads) atomicAdd(&S.base[(__ldcg(&in[i]).x >> shift) & 255u], 1u);
    __syncthreads();
    uint32_t total;
    const uint32_t excl = ctaExclusiveScan<kPlaceThreads>(S.base[tid], S.warp, &total);
    S.base[tid] = excl;
    for (uint32_t i0 = s; i0 < e; i0 += kPlaceThreads) {
      for (uint32_t w = 0; w < kPlaceThreads / 32; ++w) S.count[w][tid] = 0;
      __syncthreads();
      const uint32_t i = i0 + tid;
      const uint2 m = i < e ? __ldcg(&in[i]) : make_uint2(0u, 0u);
      const uint32_t d = i < e ? (m.x >> shift) & 255u : 256u;
      const uint32_t peers = __match_any_sync(0xFFFFFFFFu, d);
      const uint32_t rank = (uint32_t)__popc(peers & ((1u << lane) - 1u));
      if (d < 256u && rank == 0u) S.count[warp][d] = (uint16_t)__popc(peers);
      __syncthreads();
      if (d < 256u) {
        uint32_t dst = S.base[d] + rank;
        for (uint32_t w = 0; w < warp; ++w) dst += S.count[w][d];
        if (s + dst < e) out[s + dst] = m;
      }
      __syncthreads();
      uint32_t add = 0;
      for (uint32_t w = 0; w < kPlaceThreads / 32; ++w) add += S.count[w][tid];
      S.base[tid] += add;
    }
    __threadfence_block();
    __syncthreads();
  }
  for (uint32_t i = s + tid; i < e; i += kPlaceThreads) {
    const uint2 m = __ldcg(&buf[from][i]);
    A.members[i] = make_uint4(m.x, m.y, s, key);
  }
  __syncthreads();
}

// kGiantTile agents in id order, put behind the earlier tiles' in their giant
// cells: one pass of a stable partition, the tiles' counts handed on as in the
// radix sort.  scratch[0] holds (giant cell or none, slot) by agent id.
__device__ void placeGiantTile(const OrderArgs& A, CrowdShared& S, uint32_t tile, uint32_t giants) {
  constexpr uint32_t kItems = kGiantTile / kPlaceThreads, kNone = kGiants;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t first = tile * kGiantTile + warp * (32u * kItems) + lane;
  for (uint32_t w = 0; w < kPlaceThreads / 32; ++w) S.count[w][tid] = 0;
  __syncthreads();
  uint32_t at[kItems];  // the cell, and the place among the warp's agents of that cell above it
#pragma unroll
  for (uint32_t q = 0; q < kItems; ++q) {
    const uint32_t id = first + q * 32u;
    const uint32_t g0 = id < A.n ? __ldcg(&A.scratch[0][id]).x : kNone;
    const uint32_t g = g0 < giants ? g0 : kNone;
    const uint32_t peers = __match_any_sync(0xFFFFFFFFu, g);
    const uint32_t leader = (uint32_t)__ffs(peers) - 1u;
    uint32_t before = 0;
    if (lane == leader && g != kNone) {
      before = S.count[warp][g];
      S.count[warp][g] = (uint16_t)(before + (uint32_t)__popc(peers));
    }
    before = __shfl_sync(0xFFFFFFFFu, before, leader);
    at[q] = g | (before + (uint32_t)__popc(peers & ((1u << lane) - 1u))) << 16;
    __syncwarp();
  }
  __syncthreads();
  if (tid < giants) {
    uint32_t mine = 0;
    for (uint32_t w = 0; w < kPlaceThreads / 32; ++w) {
      const uint32_t c = S.count[w][tid];
      S.count[w][tid] = (uint16_t)mine;
      mine += c;
    }
    uint32_t* status = A.giantStatus + tid;
    uint32_t before = 0;
    if (tile > 0) {
      stRelaxed(&status[(size_t)tile * kGiants], kLookAgg | mine);
      // earlier tiles were claimed earlier: their blocks run, and publish
      int p = (int)tile - 1;
      uint32_t spins = 0;
      const bool stalled = tile == A.wait.stallTile;
      for (bool done = false; !done;) {
        constexpr int kAhead = 4;
        uint32_t v[kAhead];
#pragma unroll
        for (int q = 0; q < kAhead; ++q)
          v[q] = p >= q ? (stalled ? 0u : ldRelaxed(&status[(size_t)(p - q) * kGiants])) : kLookInc;
        int used = 0;
#pragma unroll
        for (int q = 0; q < kAhead; ++q) {
          const uint32_t f = v[q] & kLookMask;
          if (done || used < q || f == 0u) continue;
          before += v[q] & kLookVal;
          done = f == kLookInc;
          ++used;
        }
        p -= used;
        if (!done && used < kAhead && ++spins > A.wait.spinLimit) {
          atomicOr(A.errWord, kDevErrLookback);
          break;
        }
      }
    }
    stRelaxed(&status[(size_t)tile * kGiants], kLookInc | ((before + mine) & kLookVal));
    S.base[tid] = S.start[tid] + before;
  }
  __syncthreads();
#pragma unroll
  for (uint32_t q = 0; q < kItems; ++q) {
    const uint32_t id = first + q * 32u, g = at[q] & 0xFFFFu;
    if (g == kNone) continue;
    const uint32_t p = S.base[g] + S.count[warp][g] + (at[q] >> 16);
    if (p < S.end[g]) A.members[p] = make_uint4(id, __ldcg(&A.scratch[0][id]).y, S.start[g], S.cell[g]);
  }
  __syncthreads();
}

// A step with crowded cells: the blocks claim pieces of work in order.  First
// the places of 256 slots each, as in the other steps, but the agents of giant
// cells go to an array by id; then tiles of that array; then a crowded cell each.
// A piece waits for earlier ones only, and those are with blocks that run.
__device__ __noinline__ void placeCrowded(const OrderArgs& A, CrowdShared& S, uint32_t placeItems, uint32_t crowded, uint32_t giants) {
  const uint32_t tid = threadIdx.x;
  giants = min(giants, kGiants);
  crowded = min(crowded, bigCellCap(A.n));
  if (tid < giants) {
    const uint32_t c = A.giantCells[tid];
    S.cell[tid] = c;
    S.start[tid] = A.cellStart[c];
    S.end[tid] = A.cellEnd[c];
  }
  const uint32_t tiles = giants ? (A.n + kGiantTile - 1) / kGiantTile : 0u;
  for (;;) {
    __syncthreads();
    if (tid == 0) S.item = atomicAdd(&A.words[kOrderWordItem], 1u);
    __syncthreads();
    const uint32_t item = S.item;
    if (item >= placeItems + tiles + crowded) return;
    if (item < placeItems) {
      for (uint32_t w = item * kPlaceThreads + tid; w < tiles * kGiants; w += placeItems * kPlaceThreads) A.giantStatus[w] = 0u;
      const uint32_t j = item * kPlaceThreads + tid;
      if (j < A.n) {
        const uint2 kp = A.cellPlace[j];
        const uint32_t id = A.id[j], s = A.cellStart[kp.x], p = s + kp.y;
        uint32_t g = kGiants;
        if (giants && A.cellEnd[kp.x] - s > giantLimit(A.n))
          for (uint32_t k = 0; k < giants; ++k)
            if (S.cell[k] == kp.x) g = k;
        if (giants && id < A.n) A.scratch[0][id] = make_uint2(g, j);
        if (s != kEmpty && p < A.n) {
          if (g == kGiants) A.members[p] = make_uint4(id, j, s, kp.x);
        } else {
          atomicOr(A.errWord, kDevErrOrder);
        }
      }
      __threadfence();
      __syncthreads();
      if (tid == 0) atomicAdd(&A.words[kOrderWordDone], 1u);
      continue;
    }
    if (tid == 0) {
      uint32_t spins = 0;
      while (ldRelaxed(&A.words[kOrderWordDone]) < placeItems)
        if (++spins > A.wait.spinLimit) {
          atomicOr(A.errWord, kDevErrLookback);
          break;
        }
    }
    __syncthreads();
    __threadfence();
    if (item < placeItems + tiles) {
      placeGiantTile(A, S, item - placeItems, giants);
    } else {
      const uint32_t c = A.bigCells[item - placeItems - tiles];
      const uint32_t s = A.cellStart[c], e = A.cellEnd[c];
      if (s < e && e <= A.n) sortBigCell(A, S, s, e, c);
    }
  }
}

template <bool CHAIN>
__global__ void __launch_bounds__(kPlaceThreads, 8) placeKernel(const __grid_constant__ OrderArgs A, uint32_t blocks) {
  __shared__ CrowdShared sCrowd;
  chainBegin();
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  // (the counts of crowded cells arrive beside the loads that most steps need)
  static_assert(kOrderWordGiant == kOrderWordBig + 1 && kOrderWordBig % 2 == 0, "read as a pair");
  const uint2 crowds = *reinterpret_cast<const uint2*>(&A.words[kOrderWordBig]);
  uint2 kp = make_uint2(0u, 0u);
  uint32_t id = 0, s = 0;
  if (j < A.n) {
    kp = ldStep<CHAIN>(&A.cellPlace[j]);
    id = ldStep<CHAIN>(&A.id[j]);
    s = ldStep<CHAIN>(&A.cellStart[kp.x]);
  }
  if ((crowds.x | crowds.y) != 0u) {
    placeCrowded(A, sCrowd, blocks, crowds.x, crowds.y);
    return;
  }
  if (j < A.n) {
    const uint32_t p = s + kp.y;
    if (s != kEmpty && p < A.n) A.members[p] = make_uint4(id, j, s, kp.x);
    else atomicOr(A.errWord, kDevErrOrder);
  }
}

}  // namespace

// Cells per tile: 256 (1 a thread), 512, 1024 (256 threads) or 8192 (1024 threads of 8).
static uint32_t cellScanTile(uint32_t numCells) {
  for (uint32_t items = 1; items <= 4; items *= 2)
    if ((numCells + 256u * items - 1) / (256u * items) <= kCellScanTilesTarget) return 256u * items;
  return 8192u;
}
uint32_t orderCellTiles(uint32_t numCells) {
  const uint32_t tile = cellScanTile(numCells);
  return (numCells + tile - 1) / tile;
}

cudaError_t launchOrderCount(const OrderArgs& A, cudaStream_t st) {
  if (A.n == 0) return cudaSuccess;
  const uint32_t tiles = orderCellTiles(A.numCells);
  return launchChainedOr(A.n, countKernel<true>, countKernel<false>, (std::max(A.n, tiles) + 255) / 256, 256, 0, st, A, tiles);
}

cudaError_t launchOrderPlace(const OrderArgs& A, cudaStream_t st) {
  if (A.n == 0) return cudaSuccess;
  const uint32_t tiles = orderCellTiles(A.numCells);
  cudaError_t e;
  switch (cellScanTile(A.numCells)) {
    case 256: e = launchChained(A.n, cellScanKernel<256, 1>, tiles, 256, 0, st, A); break;
    case 512: e = launchChained(A.n, cellScanKernel<256, 2>, tiles, 256, 0, st, A); break;
    case 1024: e = launchChained(A.n, cellScanKernel<256, 4>, tiles, 256, 0, st, A); break;
    default: e = launchChained(A.n, cellScanKernel<1024, 8>, tiles, 1024, 0, st, A); break;
  }
  if (e != cudaSuccess) return e;
  const uint32_t blocks = (A.n + kPlaceThreads - 1) / kPlaceThreads;
  return launchChainedOr(A.n, placeKernel<true>, placeKernel<false>, blocks, kPlaceThreads, 0, st, A, blocks);
}

}  // namespace brt
