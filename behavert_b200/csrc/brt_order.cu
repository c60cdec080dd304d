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
// the reorder.  Cells of more than kRankLimit agents, where comparing all pairs
// would not be, are sorted by id by placeKernel's last block.
//
// The kernels are bound by latency (small worlds) or by their scattered 4 to 16
// byte accesses (large ones).  Measured, us of a warm step for all launches
// before the flock kernel, against repairing the previous order (mark, cell scan,
// place, with the hash and radix launches there but gated off): 4,096 agents 13.0
// against 29; 100,003: 17.7 against 38; 1,048,576 with 8 features: 65 against 87;
// 1,024 flocks, 10.2 M agents: 385 against 550.  After a changed state, where the
// radix sort ran: 13 against 30 (4,096), 65 against 108 (1,048,576).
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
      const uint32_t b = atomicAdd(&A.words[kOrderWordBig], 1u);
      if (b < bigCellCap(A.n)) A.bigCells[b] = c0 + k;
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

// One crowded cell's members, sorted by id: a stable radix sort on 8-bit
// digits by one CTA of kPlaceThreads threads, 256 members at a time, between
// members (id, slot) and the pair buffers.
__device__ void sortBigCell(const OrderArgs& A, uint32_t s, uint32_t e, uint32_t key) {
  __shared__ uint32_t sBase[256];
  __shared__ uint32_t sCount[kPlaceThreads / 32][256];
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  for (uint32_t i = s + tid; i < e; i += kPlaceThreads) {
    const uint4 m = __ldcg(&A.members[i]);
    A.scratch[0][i] = make_uint2(m.x, m.y);
  }
  uint32_t from = 0;
  for (uint32_t shift = 0; shift < 32u && (A.n - 1u) >> shift; shift += 8u, from ^= 1u) {
    const uint2* in = A.scratch[from];
    uint2* out = A.scratch[from ^ 1u];
    sBase[tid] = 0u;
    __syncthreads();
    for (uint32_t i = s + tid; i < e; i += kPlaceThreads) atomicAdd(&sBase[(__ldcg(&in[i]).x >> shift) & 255u], 1u);
    __syncthreads();
    __shared__ uint32_t sWarp[kPlaceThreads / 32 + 1];
    uint32_t total;
    const uint32_t excl = ctaExclusiveScan<kPlaceThreads>(sBase[tid], sWarp, &total);
    sBase[tid] = excl;
    for (uint32_t i0 = s; i0 < e; i0 += kPlaceThreads) {
      for (uint32_t w = 0; w < kPlaceThreads / 32; ++w) sCount[w][tid] = 0u;
      __syncthreads();
      const uint32_t i = i0 + tid;
      const uint2 m = i < e ? __ldcg(&in[i]) : make_uint2(0u, 0u);
      const uint32_t d = i < e ? (m.x >> shift) & 255u : 256u;
      const uint32_t peers = __match_any_sync(0xFFFFFFFFu, d);
      const uint32_t rank = (uint32_t)__popc(peers & ((1u << lane) - 1u));
      if (d < 256u && rank == 0u) sCount[warp][d] = (uint32_t)__popc(peers);
      __syncthreads();
      if (d < 256u) {
        uint32_t dst = sBase[d] + rank;
        for (uint32_t w = 0; w < warp; ++w) dst += sCount[w][d];
        if (s + dst < e) out[s + dst] = m;
      }
      __syncthreads();
      uint32_t add = 0;
      for (uint32_t w = 0; w < kPlaceThreads / 32; ++w) add += sCount[w][tid];
      sBase[tid] += add;
    }
    __threadfence_block();
    __syncthreads();
  }
  for (uint32_t i = s + tid; i < e; i += kPlaceThreads) {
    const uint2 m = __ldcg(&A.scratch[from][i]);
    A.members[i] = make_uint4(m.x, m.y, s, key);
  }
  __syncthreads();
}

template <bool CHAIN>
__global__ void __launch_bounds__(kPlaceThreads) placeKernel(OrderArgs A, uint32_t blocks) {
  __shared__ bool sLast;
  chainBegin();
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t big = A.words[kOrderWordBig];
  if (j < A.n) {
    const uint2 kp = ldStep<CHAIN>(&A.cellPlace[j]);
    const uint32_t id = ldStep<CHAIN>(&A.id[j]);
    const uint32_t s = ldStep<CHAIN>(&A.cellStart[kp.x]);
    const uint32_t p = s + kp.y;
    if (s != kEmpty && p < A.n) A.members[p] = make_uint4(id, j, s, kp.x);
    else atomicOr(A.errWord, kDevErrOrder);
  }
  if (big == 0u) return;
  // crowded cells: the last block sorts them once every member is there
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) sLast = atomicAdd(&A.words[kOrderWordDone], 1u) == blocks - 1u;
  __syncthreads();
  if (!sLast) return;
  __threadfence();
  for (uint32_t b = 0; b < min(big, bigCellCap(A.n)); ++b) {
    const uint32_t c = __ldcg(&A.bigCells[b]);
    const uint32_t s = __ldcg(&A.cellStart[c]), e = __ldcg(&A.cellEnd[c]);
    if (s < e && e <= A.n) sortBigCell(A, s, e, c);
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
