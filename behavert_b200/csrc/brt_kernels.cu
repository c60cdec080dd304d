// brt_kernels.cu -- the per-step pipeline kernels.
//
// Data layout in HBM (N agents over all flocks, C cells over all flocks):
//   canonical state  posA/fwdA/accA float4[N], featA float[N*Fs], idA u32[N]
//                    in the sorted order of the previous step (slot i holds
//                    agent idA[i]); each flock owns a fixed slot range;
//   sorted state     posS/fwdS/accS/featS/idS, the reordered copy the
//                    neighbour pass reads;
//   pairs[2]         (cell key, previous slot) uint2[N], sort ping-pong;
//   cellStart/End    u32[C], 0xFFFFFFFF when empty;
//   similarityStats  float4[N] in agent-id order (only the agent itself
//                    reads it, so it never moves).
//   members          uint4[N], the cells' agents before they are ranked by id
// One step: the order (brt_order.cu: count, cell scan, place; or hashKernel and
// the onesweep passes) -> reorderKernel -> flock kernel.
#include "brt_agent.cuh"
#include "brt_kernels.cuh"

#include <algorithm>

namespace brt {

// ---------------------------------------------------------------------------
// genCalcHashD (envgrid3d_kernel.cu:55-68): key = cellBase + cell hash of the
// agent's position, written at the agent's id so the sort input is in
// agent-id order (the reference hashes the id-ordered position array, and its
// stable sort breaks ties by id).  The value is the agent's current slot.
// The kernel also builds the digit histograms of every sort pass, clears the
// cell ranges and resets the sort's look-back state.
__global__ void __launch_bounds__(256) hashKernel(HashArgs A) {
  extern __shared__ uint32_t sHist[];
  const uint32_t histWords = A.passes * A.bins;
  for (uint32_t k = threadIdx.x; k < histWords; k += blockDim.x) sHist[k] = 0u;
  __syncthreads();
  const uint32_t gtid = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t gstride = gridDim.x * blockDim.x;
  for (uint32_t j = gtid; j < A.n; j += gstride) {
    const uint32_t f = A.nflocks == 1 ? 0u : flockOfSlot(A.agentBase, A.nflocks, j);
    const FlockDev& fl = A.flocks[f];
    const float4 p = __ldg(&A.pos[j]);
    const int gx = gridCoord(p.x, fl), gy = gridCoord(p.y, fl), gz = gridCoord(p.z, fl);
    const uint32_t key = fl.cellBase + ((uint32_t)gz * fl.G + (uint32_t)gy) * fl.G + (uint32_t)gx;
    const uint32_t id = __ldg(&A.id[j]);
    A.pairs[id] = make_uint2(key, j);
    for (uint32_t ps = 0; ps < A.passes; ++ps)
      atomicAdd(&sHist[ps * A.bins + ((key >> A.shift[ps]) & A.mask[ps])], 1u);
  }
  uint4* cs = reinterpret_cast<uint4*>(A.cellStart);
  uint4* ce = reinterpret_cast<uint4*>(A.cellEnd);
  const uint4 e4 = make_uint4(kEmpty, kEmpty, kEmpty, kEmpty);
  for (uint32_t c = gtid; c < A.cellWords4; c += gstride) { cs[c] = e4; ce[c] = e4; }
  for (uint32_t k = gtid; k < A.statusWords; k += gstride) A.status[k] = 0u;
  if (gtid < A.passes) A.counters[gtid] = 0u;
  if (gtid == 0 && A.stepCounter) *A.stepCounter += 1u;
  __syncthreads();
  for (uint32_t k = threadIdx.x; k < histWords; k += blockDim.x)
    if (sHist[k]) atomicAdd(&A.hist[k], sHist[k]);
}

// reorderDataFloat4 (envgrid3d_kernel.cu:110-122) for every registered
// feature in one pass with 128-bit accesses.  After the radix sort also
// genericFindCellStartD (Proximity3D_kernel.cu:54-84) extended to cellEnd, and
// the clearing of the digit histograms for the next step.  RANK, after the
// order by counting: thread i's agent is member i of its cell, in no order; its
// sorted position is the cell's first plus the members with smaller ids (the
// members of a cell of more than kRankLimit are in id order already).
template <bool RANK, bool CHAIN, bool OWN = false>
__global__ void __launch_bounds__(256) reorderKernel(ReorderArgs A) {
  chainBegin();
  const uint32_t gtid = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t gstride = gridDim.x * blockDim.x;
  if (!RANK)
    for (uint32_t k = gtid; k < A.histWords; k += gstride) A.hist[k] = 0u;
  bool outside = false;  // cell-cull gate: a position of this thread's slots lies outside its cell
  for (uint32_t t = gtid; t < A.n; t += gstride) {
    uint32_t key, ps, i = t;
    uint32_t prev = 0, next = 0;
    if constexpr (RANK) {
      const uint4 m = ldStep<CHAIN>(&A.members[t]);
      ps = m.y;
      key = m.w;
      const uint32_t s = m.z;
      // (a stale entry, left by a step whose waits ran out, must stay in bounds)
      if (ps >= A.n || key >= A.numCells || s > t) { atomicOr(A.errWord, kDevErrOrder); continue; }
      const uint32_t e = ldStep<CHAIN>(&A.cellEnd[key]);
      if (e > A.n || e <= t) { atomicOr(A.errWord, kDevErrOrder); continue; }
      if (e - s <= kRankLimit) {
        i = s;
        for (uint32_t q = s; q < e; ++q) i += ldStep<CHAIN>(&A.members[q].x) < m.x ? 1u : 0u;
      }
      A.pairsOut[i] = make_uint2(key, ps);
    } else {
      const uint2 kv = A.pairs[i];
      key = kv.x;
      ps = kv.y;
      if (ps >= A.n || key >= A.numCells) { atomicOr(A.errWord, kDevErrOrder); continue; }
      prev = i > 0 ? A.pairs[i - 1].x : kEmpty;
      next = i + 1 < A.n ? A.pairs[i + 1].x : kEmpty;
    }
    float4 pos = ldStep<CHAIN>(&A.posA[ps]);
    if constexpr (CHAIN) {  // an ordinary load is not moved across a store
      const float4 fwd = ldStep<CHAIN>(&A.fwdA[ps]), acc = ldStep<CHAIN>(&A.accA[ps]);
      const uint32_t id = ldStep<CHAIN>(&A.idA[ps]);
      A.fwdS[i] = fwd;
      A.accS[i] = acc;
      A.idS[i] = id;
    } else {
      A.fwdS[i] = ldStep<CHAIN>(&A.fwdA[ps]);
      A.accS[i] = ldStep<CHAIN>(&A.accA[ps]);
      A.idS[i] = ldStep<CHAIN>(&A.idA[ps]);
    }
    if (A.prevOut) A.prevOut[i] = ps;
    if (A.fs4) {
      // The feature norm sqrtf(sum f^2) (computeSimilarity's norma,
      // BehaviorClustering_resources.cu:164-175) is the same for every pair
      // an agent takes part in: compute it once here, in the same order.
      // It also goes into the sorted position's w (no kernel reads the w
      // of a position; integration always writes 1), so the list walk gets
      // a neighbour's norm with the neighbour's position.  OWN: flocks differ in
      // featuresCount, and an agent is compared over its flock's own columns.
      const float4* src = reinterpret_cast<const float4*>(A.featA) + (size_t)ps * A.fs4;
      float4* dst = reinterpret_cast<float4*>(A.featS) + (size_t)i * A.fs4;
      float nn = 0.0f;
      uint32_t own = 0;
      if constexpr (OWN) own = A.flocks[flockOfSlot(A.agentBase, A.nflocks, i)].F;
      float4 next;  // chained: one load ahead of the store, as above
      if constexpr (CHAIN) next = ldStep<CHAIN>(&src[0]);
      for (uint32_t q = 0; q < A.fs4; ++q) {
        float4 v;
        if constexpr (CHAIN) {
          v = next;
          if (q + 1 < A.fs4) next = ldStep<CHAIN>(&src[q + 1]);
        } else {
          v = ldStep<CHAIN>(&src[q]);
        }
        dst[q] = v;
        if constexpr (OWN) {
          if (4 * q + 0 >= own) v.x = 0.0f;
          if (4 * q + 1 >= own) v.y = 0.0f;
          if (4 * q + 2 >= own) v.z = 0.0f;
          if (4 * q + 3 >= own) v.w = 0.0f;
          reinterpret_cast<float4*>(A.featOwn)[(size_t)i * A.fs4 + q] = v;
        }
        nn += v.x * v.x;
        nn += v.y * v.y;
        nn += v.z * v.z;
        nn += v.w * v.w;
      }
      pos.w = sqrtf(nn);
    }
    if (A.cullWords && !outside) {
      const FlockDev& fl = A.flocks[A.nflocks == 1 ? 0u : flockOfSlot(A.agentBase, A.nflocks, i)];
      outside = !(pos.x >= 0.0f && pos.x <= fl.L && pos.y >= 0.0f && pos.y <= fl.L && pos.z >= 0.0f && pos.z <= fl.L);
    }
    A.posS[i] = pos;
    if (!RANK) {
      if (key != prev) A.cellStart[key] = i;
      if (key != next) A.cellEnd[key] = i + 1;
    }
  }
  if (A.cullWords) {
    // Scan variants 0 and 1 skip a neighbour cell by the distance from the
    // agent to the cell's face.  That bounds a candidate's distance only when
    // both lie in their hashed cells, which every finite position inside the
    // world does (L is a whole number of cells); a NaN position (clamped into
    // cell 0) or one outside the world (clamped into an edge cell) does not.
    // The last block to finish publishes the OR of all blocks' flags and
    // leaves the accumulator and the ticket at zero for the next launch.
    if (__syncthreads_or(outside) && threadIdx.x == 0) atomicOr(&A.cullWords[0], 1u);
    if (threadIdx.x == 0) {
      __threadfence();
      if (atomicAdd(&A.cullWords[1], 1u) == gridDim.x - 1) {
        A.cullWords[2] = atomicExch(&A.cullWords[0], 0u);
        A.cullWords[1] = 0u;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// The per-agent body shared by the fused pass (one thread per sorted slot).
struct AgentOut {
  Integrated r;
};

// Columns of an agent's features beyond its flock's own (flocks of one engine may
// differ in featuresCount, and state I/O carries every column) move with the agent.
template <bool CHAIN>
__device__ __forceinline__ void carryColumns(const float* __restrict__ featS, float* featA, uint32_t Fs, uint32_t i, uint32_t F) {
  const size_t row = (size_t)i * Fs;
  for (uint32_t k = F; k < Fs; ++k) featA[row + k] = ldStep<CHAIN>(&featS[row + k]);
}

__global__ void __launch_bounds__(256) carryColumnsKernel(const float* featS, float* featA, uint32_t Fs, const FlockDev* flocks,
                                                          const uint32_t* agentBase, uint32_t nflocks, uint32_t n) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) carryColumns<false>(featS, featA, Fs, i, flocks[flockOfSlot(agentBase, nflocks, i)].F);
}

template <bool CHAIN>
__device__ __forceinline__ void loadFeatures(const float* __restrict__ featS, uint32_t Fs, uint32_t i, uint32_t F, float* fi) {
  const float* src = featS + (size_t)i * Fs;
  for (uint32_t k = 0; k < F; ++k) fi[k] = ldStep<CHAIN>(&src[k]);
}

// The list-first kernel (option "two_pass", kNN lists above a warp, kNN and
// clustering flocks in one engine): neighbour search, flocking steering,
// clustering, obstacles, feature relaxation, integration.  Lists stay in shared memory
// ([k][thread] layout, odd stride) unless recording is on.  First-M lists
// come from the warp-cooperative windowed scan (every lane of a warp takes
// part; inactive lanes mirror the last agent read-only and leave after it),
// kNN lists (maxNeighbors above a warp) from the per-agent scan.
template <bool KNN, bool CHAIN>
__global__ void __launch_bounds__(kFusedThreads) fusedKernel(FusedArgs A) {
  extern __shared__ uint32_t sList[];
  __shared__ float4 sSegs[KNN ? 1 : kFusedThreads / 32 * kSegments];
  chainBegin();
  uint32_t i0;
  const bool active = KNN ? (i0 = blockIdx.x * blockDim.x + threadIdx.x) < A.n : agentOfLane(A.warpAgents, A.n, i0);
  if (KNN && !active) return;
  const uint32_t i = active ? i0 : A.n - 1;
  const uint32_t f = A.nflocks == 1 ? 0u : flockOfSlot(A.agentBase, A.nflocks, i);
  const FlockDev& fl = A.flocks[f];
  const float4 p4 = ldStep<CHAIN>(&A.posS[i]);
  uint32_t* list = sList + threadIdx.x;
  const uint32_t ls = blockDim.x + 1;
  uint32_t n;
  if constexpr (KNN) {
    float distL[BRT_MAX_NEIGHBORS];
    n = buildNeighborList<CHAIN, true>(i, xyz(p4), fl, A.cellStart, A.cellEnd, A.posS, list, ls, distL);
  } else {
    const f3 p = xyz(p4);
    const HomeCell home = homeCell(gridCoord(p.x, fl), gridCoord(p.y, fl), gridCoord(p.z, fl), fl);
    n = scanNeighborsCooperative<CHAIN, kCoopCachedRounds, kCoopWindowAgents>(active, i, p, home, A.flocks, f, A.cellStart,
                                                                      A.cellEnd, A.posS, sList, ls, threadIdx.x & ~31u,
                                                                      sSegs + (threadIdx.x >> 5) * kSegments);
    if (!active) return;
  }
  const float4 w4 = ldStep<CHAIN>(&A.fwdS[i]);
  const float4 a4 = ldStep<CHAIN>(&A.accS[i]);
  if (A.lists) {
    uint32_t* out = A.lists + (size_t)i * A.listStride;
    out[0] = n;
    for (uint32_t k = 0; k < n; ++k) out[1 + k] = list[k * ls];
  }
  const AgentCtx a = makeCtx(p4, w4, fl);
  f3 steer = mk3(0.f, 0.f, 0.f);
  steer = flockingSteer<CHAIN>(a, fl, list, ls, n, A.posS, A.fwdS, steer, fl.sep[0] != 0.0f, fl.ali[0] != 0.0f, fl.coh[0] != 0.0f);
  float fi[BRT_MAX_FEATUREDIM];
  float norm1 = 0.0f;
  const uint32_t F = fl.F;
  if (F) {
    loadFeatures<CHAIN>(A.featS, A.Fs, i, F, fi);
    norm1 = selfNorm(fi, F);
  }
  if (F && (fl.clus != 0.0f || fl.aclus != 0.0f)) {
    const uint32_t id = ldStep<CHAIN>(&A.idS[i]);
    float4 st = A.statsById[id];
    float sims[BRT_MAX_NEIGHBORS];
    steer = clusteringSteer<CHAIN>(a, fl, list, ls, n, A.posS, A.fwdS, fi, norm1, A.featS, A.Fs, st, sims, steer);
    A.statsById[id] = st;
  }
  if (fl.numObstacles && fl.obsW != 0.0f) steer = obstacleSteer(a, fl, A.obstacles, A.obsMask, steer);
  if (F) {
    float fo[BRT_MAX_FEATUREDIM];
    relaxFeatures<CHAIN>(fl, list, ls, n, fi, norm1, A.featS, A.Fs, fo);
    float* dst = A.featA + (size_t)i * A.Fs;
    for (uint32_t k = 0; k < F; ++k) dst[k] = fo[k];
  }
  carryColumns<CHAIN>(A.featS, A.featA, A.Fs, i, F);
  const Integrated r = integrate(a, a4, steer, A.dt, fl);
  A.posA[i] = r.pos;
  A.fwdA[i] = r.fwd;
  A.accA[i] = r.acc;
  A.idA[i] = ldStep<CHAIN>(&A.idS[i]);
}

// ---------------------------------------------------------------------------
// Stage-wise kernels (the reference's separate functionalities).

// computeNeighborhoods: every agent's list into the list array.  First-M
// lists come from the warp-cooperative windowed scan through shared memory
// (inactive lanes take part read-only), kNN lists from the per-agent scan.
template <bool KNN>
__global__ void __launch_bounds__(128) listsKernel(StageArgs A) {
  extern __shared__ uint32_t sList[];
  __shared__ float4 sSegs[KNN ? 1 : 4 * kSegments];
  uint32_t i0;
  const bool active = KNN ? (i0 = blockIdx.x * blockDim.x + threadIdx.x) < A.n : agentOfLane(A.warpAgents, A.n, i0);
  if (KNN && !active) return;
  const uint32_t i = active ? i0 : A.n - 1;
  const uint32_t f = A.nflocks == 1 ? 0u : flockOfSlot(A.agentBase, A.nflocks, i);
  const FlockDev& fl = A.flocks[f];
  uint32_t* out = A.lists + (size_t)i * A.listStride;
  const f3 p = xyz(__ldg(&A.posS[i]));
  if constexpr (KNN) {
    float distL[BRT_MAX_NEIGHBORS];
    out[0] = buildNeighborList<false, true>(i, p, fl, A.cellStart, A.cellEnd, A.posS, out + 1, 1, distL);
  } else {
    const HomeCell home = homeCell(gridCoord(p.x, fl), gridCoord(p.y, fl), gridCoord(p.z, fl), fl);
    const uint32_t ls = blockDim.x + 1;
    const uint32_t n = scanNeighborsCooperative<false, kCoopCachedRounds, kCoopWindowAgents>(
        active, i, p, home, A.flocks, f, A.cellStart, A.cellEnd, A.posS, sList, ls, threadIdx.x & ~31u,
        sSegs + (threadIdx.x >> 5) * kSegments);
    if (!active) return;
    const uint32_t* list = sList + threadIdx.x;
    for (uint32_t k = 0; k < n; ++k) out[1 + k] = list[k * ls];
    out[0] = n;
  }
}

// which: 0 separation, 1 alignment, 2 cohesion, 3 clustering, 4 obstacles
__global__ void __launch_bounds__(128) steerStageKernel(StageArgs A, int which) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= A.n) return;
  const uint32_t f = A.nflocks == 1 ? 0u : flockOfSlot(A.agentBase, A.nflocks, i);
  const FlockDev& fl = A.flocks[f];
  const uint32_t* lst = A.lists + (size_t)i * A.listStride;
  const uint32_t n = lst[0];
  const AgentCtx a = makeCtx(__ldg(&A.posS[i]), __ldg(&A.fwdS[i]), fl);
  const float4 s4 = A.steer[i];
  f3 steer = xyz(s4);
  if (which == 0 && fl.sep[0] != 0.0f) steer = flockingSteer<false>(a, fl, lst + 1, 1, n, A.posS, A.fwdS, steer, true, false, false);
  if (which == 1 && fl.ali[0] != 0.0f) steer = flockingSteer<false>(a, fl, lst + 1, 1, n, A.posS, A.fwdS, steer, false, true, false);
  if (which == 2 && fl.coh[0] != 0.0f) steer = flockingSteer<false>(a, fl, lst + 1, 1, n, A.posS, A.fwdS, steer, false, false, true);
  if (which == 3 && fl.F && (fl.clus != 0.0f || fl.aclus != 0.0f)) {
    float fi[BRT_MAX_FEATUREDIM];
    loadFeatures<false>(A.featS, A.Fs, i, fl.F, fi);
    const float norm1 = selfNorm(fi, fl.F);
    const uint32_t id = __ldg(&A.idS[i]);
    float4 st = A.statsById[id];
    float sims[BRT_MAX_NEIGHBORS];
    steer = clusteringSteer<false>(a, fl, lst + 1, 1, n, A.posS, A.fwdS, fi, norm1, A.featS, A.Fs, st, sims, steer);
    A.statsById[id] = st;
  }
  if (which == 4 && fl.numObstacles && fl.obsW != 0.0f) steer = obstacleSteer(a, fl, A.obstacles, A.obsMask, steer);
  if (which == 5) {
    // The new speed goes to this agent's own forward entry, which no other
    // thread reads in this stage; blendIntoSteeringForce adds the force.
    float speed = a.speed;
    const f3 s = avoidNeighbors(a, fl, lst + 1, 1, n, A.posS, &speed);
    A.fwdW[i] = make_float4(a.fwd.x, a.fwd.y, a.fwd.z, speed);
    steer = add3(s, steer);
  }
  if (which == 6) {
    // moveAwayFromTarget_kernel (OpenSteerWrapper_kernel.cu:185-212): flee the
    // base point, (weight * offset) / distance, nothing beyond twice the
    // radius.  The kernel's acceleration write is overwritten by its own copy
    // of the old value, so the smoothed acceleration is left as it is.  As in
    // the reference: the direct offset (no periodic image), and 0/0 for an
    // agent exactly at the base point.
    f3 s = sub3(a.pos, mk3(A.avoidBase[0], A.avoidBase[1], A.avoidBase[2]));
    const float d = len3(s);
    if (d > A.avoidBaseParams[2] * 2.0f) s = mk3(0.f, 0.f, 0.f);
    steer = add3(div3(mul3(s, A.avoidBaseParams[0]), d), steer);
  }
  A.steer[i] = make_float4(steer.x, steer.y, steer.z, 0.0f);
}

__global__ void __launch_bounds__(128) integrateStageKernel(StageArgs A, float dt) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= A.n) return;
  const uint32_t f = A.nflocks == 1 ? 0u : flockOfSlot(A.agentBase, A.nflocks, i);
  const FlockDev& fl = A.flocks[f];
  const uint32_t* lst = A.lists + (size_t)i * A.listStride;
  const uint32_t n = lst[0];
  const float4 p4 = __ldg(&A.posS[i]), w4 = __ldg(&A.fwdS[i]), a4 = __ldg(&A.accS[i]);
  const AgentCtx a = makeCtx(p4, w4, fl);
  if (fl.F) {
    float fi[BRT_MAX_FEATUREDIM], fo[BRT_MAX_FEATUREDIM];
    loadFeatures<false>(A.featS, A.Fs, i, fl.F, fi);
    const float norm1 = selfNorm(fi, fl.F);
    relaxFeatures<false>(fl, lst + 1, 1, n, fi, norm1, A.featS, A.Fs, fo);
    float* dst = A.featA + (size_t)i * A.Fs;
    for (uint32_t k = 0; k < fl.F; ++k) dst[k] = fo[k];
  }
  carryColumns<false>(A.featS, A.featA, A.Fs, i, fl.F);
  const Integrated r = integrate(a, a4, xyz(A.steer[i]), dt, fl);
  A.posA[i] = r.pos;
  A.fwdA[i] = r.fwd;
  A.accA[i] = r.acc;
  A.idA[i] = __ldg(&A.idS[i]);
}

// ---------------------------------------------------------------------------
// State I/O between agent-id order and the canonical slot order.


// All arrays of a call in one launch: thread t moves agent t's vectors and
// piece t of the features (a float4 where both sides allow it, else a float),
// so a small engine's call costs one launch instead of up to four, and a large
// one's feature accesses are 16 bytes wide (one array a launch there).
// 1,048,576 agents with 8 features: set 71 -> 48 us, get 98 -> 58; 4,096 agents:
// three launches of 2.5 us -> one of 3.
// Gather: slot i takes agent id[i]'s values (positions keep w = 1, like the
// reference's position feature; the features' padding is zero).  Scatter: agent
// id[i] gets slot i's.  A row of single floats is gathered in pieces of a float4 of
// the padded canonical row.  us of a set call, an agent a thread / a float a thread /
// so: 1,000,000 agents with 3 features 49.9 / 53.7 / 48.4, 9: 99.3 / 88.9 / 59.2;
// 4,000,000 with 3: 173 / 202 / 164, 9: 349 / 373 / 235.
template <bool GATHER, bool WIDE>
__global__ void __launch_bounds__(256) stateIoKernel(StateIoArgs A) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;  // at most 2^26 agents of 32 features
  if (t < A.n) {
    const uint32_t id = __ldg(&A.id[t]);
    const size_t from = GATHER ? id : t, to = GATHER ? t : id;
    float4 v[3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
      if (A.src[k]) v[k] = __ldg(&A.src[k][from]);
    if (GATHER) v[0].w = 1.0f;
#pragma unroll
    for (int k = 0; k < 3; ++k)
      if (A.src[k]) A.dst[k][to] = v[k];
  }
  // pieces of an agent's features: on the canonical side Fs floats, on the other F
  const uint32_t per = WIDE || GATHER ? A.Fs / 4 : A.F;
  if (t >= A.n * per) return;
  const uint32_t i = t / per, k = t - i * per;
  const uint32_t id = __ldg(&A.id[i]);
  if constexpr (WIDE) {
    const float4* src = reinterpret_cast<const float4*>(A.featSrc);
    float4* dst = reinterpret_cast<float4*>(A.featDst);
    const size_t slot = (size_t)i * (A.Fs / 4) + k, agent = (size_t)id * per + k;
    dst[GATHER ? slot : agent] = __ldg(&src[GATHER ? agent : slot]);
  } else if (GATHER) {
    const float* src = A.featSrc + (size_t)id * A.F + 4 * k;
    const uint32_t left = A.F - 4 * k;
    reinterpret_cast<float4*>(A.featDst)[(size_t)i * per + k] =
        make_float4(__ldg(src), left > 1 ? __ldg(src + 1) : 0.0f, left > 2 ? __ldg(src + 2) : 0.0f, left > 3 ? __ldg(src + 3) : 0.0f);
  } else {
    A.featDst[(size_t)id * A.F + k] = __ldg(&A.featSrc[(size_t)i * A.Fs + k]);
  }
}
__global__ void hashPairsToOutKernel(const uint2* __restrict__ pairs, const uint32_t* __restrict__ idS, uint32_t* keys, uint32_t* ids, uint32_t n) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (keys) keys[i] = pairs[i].x;
  if (ids) ids[i] = __ldg(&idS[i]);
}

// ---------------------------------------------------------------------------
// Launchers.

static inline uint32_t blocksFor(uint32_t n, uint32_t t) { return (n + t - 1) / t; }

cudaError_t launchHash(const HashArgs& A, uint32_t smBlocks, cudaStream_t st) {
  const uint32_t blocks = std::max(1u, std::min(blocksFor(A.n, 256), smBlocks));
  hashKernel<<<blocks, 256, A.passes * A.bins * 4, st>>>(A);
  return cudaGetLastError();
}
cudaError_t launchCarryColumns(const float* featS, float* featA, uint32_t Fs, const FlockDev* flocks, const uint32_t* agentBase,
                               uint32_t nflocks, uint32_t n, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  carryColumnsKernel<<<blocksFor(n, 256), 256, 0, st>>>(featS, featA, Fs, flocks, agentBase, nflocks, n);
  return cudaGetLastError();
}
cudaError_t launchReorder(const ReorderArgs& A, cudaStream_t st) {
  if (A.members) {
    const uint32_t blocks = std::max(1u, blocksFor(A.n, 256));
    if (A.featOwn)
      return launchChainedOr(A.n, reorderKernel<true, true, true>, reorderKernel<true, false, true>, blocks, 256, 0, st, A);
    return launchChainedOr(A.n, reorderKernel<true, true>, reorderKernel<true, false>, blocks, 256, 0, st, A);
  }
  const uint32_t blocks = std::max(1u, blocksFor(std::max(A.n, A.histWords), 256));
  if (A.featOwn)
    return launchChainedOr(A.n, reorderKernel<false, true, true>, reorderKernel<false, false, true>, blocks, 256, 0, st, A);
  return launchChainedOr(A.n, reorderKernel<false, true>, reorderKernel<false, false>, blocks, 256, 0, st, A);
}
cudaError_t configureFusedKernels(uint32_t Mmax) {
  const int smem = (int)((size_t)(kFusedThreads + 1) * Mmax * 4);
  const void* fns[4] = {(const void*)fusedKernel<true, false>, (const void*)fusedKernel<true, true>,
                        (const void*)fusedKernel<false, false>, (const void*)fusedKernel<false, true>};
  for (const void* fn : fns) {
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
  }
  return cudaFuncSetAttribute(listsKernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(129 * Mmax * 4));
}
namespace {
uint32_t residentWarpAgents(const void* fn, int threads, size_t smem, uint32_t n, uint32_t smCount) {
  int per = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, threads, smem) != cudaSuccess || per < 1) {
    cudaGetLastError();
    per = 1;
  }
  return warpAgentsFor(n, smCount * (uint32_t)(per * threads / 32) / 2);
}
}  // namespace
uint32_t fusedWarpAgents(uint32_t n, uint32_t Mmax, uint32_t smCount) {
  return residentWarpAgents((const void*)fusedKernel<false, false>, kFusedThreads, (size_t)(kFusedThreads + 1) * Mmax * 4, n, smCount);
}
uint32_t listsWarpAgents(uint32_t n, uint32_t Mmax, uint32_t smCount) {
  return residentWarpAgents((const void*)listsKernel<false>, 128, (size_t)129 * Mmax * 4, n, smCount);
}
cudaError_t launchFused(const FusedArgs& A, bool knn, cudaStream_t st) {
  if (A.n == 0) return cudaSuccess;
  const size_t smem = (size_t)(kFusedThreads + 1) * A.Mmax * 4;
  if (knn)
    return launchChainedOr(A.n, fusedKernel<true, true>, fusedKernel<true, false>, blocksFor(A.n, kFusedThreads), kFusedThreads,
                           smem, st, A);
  return launchChainedOr(A.n, fusedKernel<false, true>, fusedKernel<false, false>,
                         blocksFor(A.n, kFusedThreads / 32 * A.warpAgents), kFusedThreads, smem, st, A);
}
cudaError_t launchLists(const StageArgs& A, bool knn, cudaStream_t st) {
  if (A.n == 0) return cudaSuccess;
  if (knn) listsKernel<true><<<blocksFor(A.n, 128), 128, 0, st>>>(A);
  else listsKernel<false><<<blocksFor(A.n, 128 / 32 * A.warpAgents), 128, (size_t)129 * (A.listStride - 1) * 4, st>>>(A);
  return cudaGetLastError();
}
// Registered per-agent arrays of `words` 32-bit words: slot i of dst takes
// slot index[i * stride] of src (gather), or slot i of src goes to slot
// index[i] of dst (scatter); one thread per word.
__global__ void gatherWordsKernel(const uint32_t* __restrict__ src, const uint32_t* __restrict__ index, uint32_t stride,
                                  uint32_t* __restrict__ dst, uint32_t words, uint32_t n) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (size_t)n * words) return;
  const size_t i = t / words, k = t - i * words;
  const uint32_t from = __ldg(&index[i * stride]);
  dst[t] = from < n ? src[(size_t)from * words + k] : 0u;  // a corrupted step's stale index reads nothing
}
__global__ void scatterWordsKernel(const uint32_t* __restrict__ src, const uint32_t* __restrict__ index,
                                   uint32_t* __restrict__ dst, uint32_t words, uint32_t n) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (size_t)n * words) return;
  const size_t i = t / words, k = t - i * words;
  dst[(size_t)__ldg(&index[i]) * words + k] = src[t];
}
cudaError_t launchGatherWords(const uint32_t* src, const uint32_t* index, uint32_t stride, uint32_t* dst, uint32_t words,
                              uint32_t n, cudaStream_t st) {
  const size_t total = (size_t)n * words;
  if (total == 0) return cudaSuccess;
  gatherWordsKernel<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(src, index, stride, dst, words, n);
  return cudaGetLastError();
}
cudaError_t launchScatterWords(const uint32_t* src, const uint32_t* index, uint32_t* dst, uint32_t words, uint32_t n,
                               cudaStream_t st) {
  const size_t total = (size_t)n * words;
  if (total == 0) return cudaSuccess;
  scatterWordsKernel<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(src, index, dst, words, n);
  return cudaGetLastError();
}

cudaError_t launchSteerStage(const StageArgs& A, int which, cudaStream_t st) {
  if (A.n == 0) return cudaSuccess;
  steerStageKernel<<<blocksFor(A.n, 128), 128, 0, st>>>(A, which);
  return cudaGetLastError();
}
cudaError_t launchIntegrateStage(const StageArgs& A, float dt, cudaStream_t st) {
  if (A.n == 0) return cudaSuccess;
  integrateStageKernel<<<blocksFor(A.n, 128), 128, 0, st>>>(A, dt);
  return cudaGetLastError();
}
namespace {
cudaError_t launchStateIoArrays(const StateIoArgs& A, bool gather, cudaStream_t st) {
  const bool wide = A.featSrc && A.F % 4 == 0 && (((uintptr_t)A.featSrc | (uintptr_t)A.featDst) & 15u) == 0;
  StateIoArgs B = A;
  if (!B.featSrc) B.F = B.Fs = 0;
  const size_t pieces = (size_t)B.n * (wide || gather ? B.Fs / 4 : B.F);
  const uint32_t blocks = (uint32_t)((std::max<size_t>(B.n, pieces) + 255) / 256);
  if (gather && wide) stateIoKernel<true, true><<<blocks, 256, 0, st>>>(B);
  else if (gather) stateIoKernel<true, false><<<blocks, 256, 0, st>>>(B);
  else if (wide) stateIoKernel<false, true><<<blocks, 256, 0, st>>>(B);
  else stateIoKernel<false, false><<<blocks, 256, 0, st>>>(B);
  return cudaGetLastError();
}
// Above this many agents each array takes a launch of its own: three streams
// of scattered 16-byte accesses at once then cost more than the launches save.
// us of a get call together / apart, no features and 8: 262,144 agents 7.9 / 15.7
// and 10.2 / 20.3, 600,000: 12.6 / 18.7 and 18.1 / 31.2, 1,000,000: 20.4 / 30.6 and
// 61.9 / 57.4; 10.2 M: 415 / 294.  (Below about 400,000 the launches' own host time
// decides.)  The line is on the safe side of where the two cross.
constexpr uint32_t kStateIoTogether = 1u << 18;
}  // namespace
cudaError_t launchStateIo(const StateIoArgs& A, bool gather, cudaStream_t st) {
  if (A.n == 0) return cudaSuccess;
  if (A.n > kStateIoTogether) {
    // one array a launch
    StateIoArgs one = A;
    for (int k = 0; k < 4; ++k) {
      for (int c = 0; c < 3; ++c) one.src[c] = c == k ? A.src[c] : nullptr;
      one.featSrc = k == 3 ? A.featSrc : nullptr;
      if (k < 3 ? !one.src[k] : !one.featSrc) continue;
      const cudaError_t e = launchStateIoArrays(one, gather, st);
      if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
  }
  return launchStateIoArrays(A, gather, st);
}
cudaError_t launchHashPairsOut(const uint2* pairs, const uint32_t* idS, uint32_t* keys, uint32_t* ids, uint32_t n, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  hashPairsToOutKernel<<<blocksFor(n, 256), 256, 0, st>>>(pairs, idS, keys, ids, n);
  return cudaGetLastError();
}

}  // namespace brt
