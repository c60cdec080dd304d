// brt_internal.cuh -- shared declarations of the CUDA library (not installed).
//
// The whole library is compiled with --fmad=false and IEEE division / square
// root, so every float + - * / sqrt below is one correctly rounded operation
// in the order written.  That is the same operation sequence the reference's
// device functions spell out (Core/common_resources.cu, the *_resources.cu
// files of the plugins), so results are reproducible bit for bit by a host
// build of the same sequence.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>
#include <cstdio>
#include <string>

#include "../../include/behavert_b200.h"

#include <nvtx3/nvToolsExt.h>

namespace brt {

constexpr uint32_t kEmpty = 0xFFFFFFFFu;
// Device error word bits (set by kernels, read by brt_engine_check_device_error).
constexpr uint32_t kDevErrLookback = 1u;   // onesweep look-back spin limit hit
constexpr uint32_t kDevErrCapacity = 2u;   // a per-kernel capacity check fired
constexpr uint32_t kDevErrOrder = 4u;      // pipeline invariant violated

// Per-flock parameters as the kernels read them (one entry per flock).
struct FlockDev {
  // geometry: periodic cube [0, L)^3, G cells per side of size cell
  uint32_t G, C, cellBase, agentBase, n;
  float L, cell;
  // Proximity3D
  float radius;
  float r2thr;          // d2 <= r2thr  <=>  !(sqrtf(d2) > radius)
  uint32_t M, maxPerCell;
  int32_t useKnn;
  // OpenSteerWrapper
  float maxSpeed, maxForce, mass, minR;
  float sep[3], ali[3], coh[3];
  int32_t use2D;
  // BehaviorClustering
  uint32_t F;
  float relax;
  float clus, aclus;
  float simStats[3];
  float avgCtl;
  // obstacles
  uint32_t numObstacles;
  float obsW;
  uint32_t obsBase;     // first entry in the engine-wide obstacle table
  float invCell;        // 1 / cell when cell is a power of two (exact), else 0
  // inBoidNeighborhood as exact squared-distance tests:
  //   dist < minR  <=>  d2 < minT,   dist > maxR_b  <=>  d2 > maxT_b
  float minT, sepT, aliT, cohT;
  // Square of -max(cosMaxAngle) when every cosMaxAngle < -1, else 0: for an
  // agent with |forward|^2 * 1.002 below it, every finite cosine passes the
  // angle test, which then only rejects NaN (a zero offset).
  float cosBound2;
  // SchoolingParams (0: flocking law; 1: animateSchool; 2: split path)
  int32_t school;
  float schTheta, schRr, schRp, schEta, schWa, schWo, schS, schRand;
  uint32_t schSeed;
};

// ---------------------------------------------------------------------------
// float3 helpers in the reference's operation order (cutil_math semantics,
// normalize = v * (1 / sqrtf(dot(v, v)))).
struct f3 { float x, y, z; };
__host__ __device__ __forceinline__ f3 mk3(float x, float y, float z) { f3 r; r.x = x; r.y = y; r.z = z; return r; }
__host__ __device__ __forceinline__ f3 add3(f3 a, f3 b) { return mk3(a.x + b.x, a.y + b.y, a.z + b.z); }
__host__ __device__ __forceinline__ f3 sub3(f3 a, f3 b) { return mk3(a.x - b.x, a.y - b.y, a.z - b.z); }
__host__ __device__ __forceinline__ f3 mul3(f3 a, float s) { return mk3(a.x * s, a.y * s, a.z * s); }
__host__ __device__ __forceinline__ f3 div3(f3 a, float s) { return mk3(a.x / s, a.y / s, a.z / s); }
__host__ __device__ __forceinline__ float dot3(f3 a, f3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__host__ __device__ __forceinline__ float len3(f3 a) { return sqrtf(dot3(a, a)); }
__host__ __device__ __forceinline__ f3 normalize3(f3 v) { float inv = 1.0f / sqrtf(dot3(v, v)); return mul3(v, inv); }
__host__ __device__ __forceinline__ float clampf(float f, float a, float b) { return fmaxf(a, fminf(f, b)); }
__host__ __device__ __forceinline__ f3 xyz(float4 v) { return mk3(v.x, v.y, v.z); }

// envgrid3d_resources.cu:60-84 with origin 0 and clamping to the grid.
// x / cell for a power-of-two cell is computed as x * (1 / cell): the
// reciprocal is exact, and the product and the quotient are the correctly
// rounded values of the same real number, so they agree bit for bit (NaN,
// infinities and subnormals included) at a fraction of an IEEE division.
__device__ __forceinline__ int gridCoordQuotient(float x, const FlockDev& fl) {
  int g = (int)floorf(x / fl.cell);
  return max(0, min(g, (int)fl.G - 1));
}
__device__ __forceinline__ int gridCoord(float x, const FlockDev& fl) {
  const float u = fl.invCell != 0.0f ? x * fl.invCell : x / fl.cell;
  int g = (int)floorf(u);
  return max(0, min(g, (int)fl.G - 1));
}

// Neighbour cell through offset o from home coordinate g, with its image shift.
__device__ __forceinline__ int wrapCoord(int c, uint32_t G) {
  return c < 0 ? c + (int)G : (c >= (int)G ? c - (int)G : c);
}
// Image shift of the neighbour cell g + o (o in {-1, 0, 1}) seen from home
// coordinate g: -L when it wraps below 0, +L when it wraps past G - 1.
// Written on the unwrapped coordinate: the equivalent form
// (o < 0 && g == 0) ? -L : ((o > 0 && g == G - 1) ? L : 0) was compiled
// wrongly for sm_100a at -O3 (nvcc 12.9) when o came from lane arithmetic
// (it returned +L for g = 0, o = +1); a probe checked this form over every
// (g, o) at the seams and in the interior.
__device__ __forceinline__ float imageShift(int g, int o, uint32_t G, float L) {
  const int c = g + o;
  return c < 0 ? -L : (c >= (int)G ? L : 0.0f);
}

// Image shift of a listed neighbour from the two cell coordinates (the
// neighbour is at most one cell away modulo the wrap, and G >= 3): a cell
// difference above 1 means the neighbour is across the lower seam, below -1
// across the upper one.  Written on the difference for the same reason as
// imageShift (the comparison form miscompiled in the same probe).
__device__ __forceinline__ float imageShiftCells(int gi, int gj, uint32_t G, float L) {
  (void)G;
  const int d = gj - gi;
  return d > 1 ? -L : (d < -1 ? L : 0.0f);
}

// Relaxed GPU-scope load and store: the look-back words of the radix passes
// and of the cell scan, polled and published across CTAs.
__device__ __forceinline__ uint32_t ldRelaxed(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void stRelaxed(uint32_t* p, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Flock of a sorted slot (flocks own contiguous slot ranges).
// A cell's sorted-slot range [start, end) as the neighbour scans use it:
// empty unless it lies inside the flock's slots.  A well-formed step always
// passes; after a corrupted one (a look-back wait that ran out, reported
// through the device error word) the words can be stale or torn, and a scan
// must never follow them out of the arrays.
__device__ __forceinline__ bool usableRange(const FlockDev& fl, uint32_t start, uint32_t end) {
  return start != kEmpty && end > start && start >= fl.agentBase && end <= fl.agentBase + fl.n;
}

__device__ __forceinline__ uint32_t flockOfSlot(const uint32_t* __restrict__ agentBase, uint32_t nflocks, uint32_t slot) {
  uint32_t lo = 0, hi = nflocks;  // agentBase has nflocks+1 entries
  while (hi - lo > 1) {
    uint32_t mid = (lo + hi) >> 1;
    if (__ldg(&agentBase[mid]) <= slot) lo = mid; else hi = mid;
  }
  return lo;
}

// The same, all lanes of a warp searching from its first lane's slot: the
// loads are the warp's, and few slots then lie in a later flock.
__device__ __forceinline__ uint32_t flockOfSlotInWarp(const uint32_t* __restrict__ agentBase, uint32_t nflocks, uint32_t slot) {
  uint32_t f = flockOfSlot(agentBase, nflocks, slot & ~31u);
  while (f + 1 < nflocks && __ldg(&agentBase[f + 1]) <= slot) ++f;
  return f;
}

// The kernels of a step follow one another on a stream, each reading what the
// one before wrote.  In a small engine launchChained has a kernel's blocks set
// up while the previous kernel still runs; they wait here, before they touch any
// memory, until it has finished and its writes are visible, and then let the
// next kernel's blocks be set up.  That takes most of a launch gap out of each of
// a step's five launches: 500 agents 25.3 -> 23.7 us a step, 4,096: 27.2 -> 25.9.
// Every block of a chained kernel calls this first, so a kernel's end means that
// all earlier ones ended.  Not in larger engines: blocks that wait take the SM
// slots that are free early, so the ones that work later are unevenly spread and
// other streams' blocks find no room (65,536 agents 55 -> 65 us; three kNN engines
// of 262,144 in turn 396 -> 697).  us a step plain / chained, alone and three engines
// in turn: 5,000 agents 38.6 / 36.4 and 14.7 / 14.3, with 8 features 46.5 / 44.2 and
// 18.2 / 17.8; 7,000: 38.8 / 37.1 and 15.5 / 15.2, 47.3 / 45.1 and 19.3 / 19.3; 16,000:
// 39.7 / 40.5 and 16.3 / 17.8, 47.6 / 49.0 and 20.6 / 21.9.  The line is a little
// below where engines side by side gain nothing more.
//
// A chained kernel reads what the step's other kernels write with ordinary loads
// (ldStep<true>), not with __ldg: a non-coherent load asks for memory that nothing
// writes while the kernel exists, and a chained kernel's blocks exist while their
// predecessor writes; the compiler may also move such a load up past the wait, which
// orders ordinary accesses only.  Kernels that also run unchained come in two
// instantiations: with ordinary loads everywhere the 1,024-flock batch's step takes
// 3,780 instead of 3,656 us (place +20%, reorder +11%, flock +3%: loads the compiler
// may not move across stores and votes).  __ldg stays for the tables that only the
// host and kernels in full order write (agentBase, obstacles, obsMask, tiles).
constexpr uint32_t kChainAgents = 5000;
template <bool CHAIN, class T>
__device__ __forceinline__ T ldStep(const T* p) {
  if constexpr (CHAIN) return *p;
  else return __ldg(p);
}
__device__ __forceinline__ void chainBegin() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
// A kernel that reads nothing of a step by ldStep, chained or not.
template <class... P, class... Q>
inline cudaError_t launchChained(uint32_t agents, void (*kernel)(P...), dim3 grid, uint32_t block, size_t smem, cudaStream_t st,
                                 Q&&... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = agents <= kChainAgents ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}
// The chained instantiation of a kernel in a small engine, else the plain one.
template <class... P, class... Q>
inline cudaError_t launchChainedOr(uint32_t agents, void (*chained)(P...), void (*plain)(P...), dim3 grid, uint32_t block,
                                   size_t smem, cudaStream_t st, Q&&... args) {
  return launchChained(agents, agents <= kChainAgents ? chained : plain, grid, block, smem, st, args...);
}
// Never chained: a launch in full order.
template <class... P, class... Q>
inline cudaError_t launchPlain(void (*kernel)(P...), dim3 grid, uint32_t block, size_t smem, cudaStream_t st, Q&&... args) {
  return launchChained(kChainAgents + 1, kernel, grid, block, smem, st, args...);
}

// ---------------------------------------------------------------------------
// Sort plan shared by the engine and the standalone entry point.
// Bound of every decoupled look-back wait (onesweep passes, the cell scan
// of the order by counting): polls of a predecessor's unpublished status word
// before the tile gives up, records kDevErrLookback and goes on (the host
// then reports BRT_ERR_TIMEOUT).  About a second at the default.
// stallTile names one tile whose look-back polls as if its predecessor never
// published (a status word that nothing sets), so that tests can make a wait
// run out on purpose; kNoStallTile in normal use.
constexpr uint32_t kDefaultSpinLimit = 1u << 21;
constexpr uint32_t kNoStallTile = 0xFFFFFFFFu;
struct LookbackWait {
  uint32_t spinLimit = kDefaultSpinLimit;
  uint32_t stallTile = kNoStallTile;
};

struct SortPlan {
  uint32_t n = 0, bits = 0, passes = 0, digitBits = 0, bins = 0, tiles = 0;
  uint32_t shift[4] = {0, 0, 0, 0};
  LookbackWait wait;
};
constexpr uint32_t kSortThreads = 512;
// Items a thread ranks per tile of 4096 pairs: 8, or 4 of 2048 for 9-bit digits,
// whose per-warp digit counters would not fit beside a 4096-pair tile in shared
// memory.  A tile's time is mostly its chain of rankings (a match and a counter
// update an item), so 512 threads of 8 beat 256 of 16: 300,000 pairs of 24 bits
// 74 -> 68 us a call, 8,000,000: 387 -> 370.
__host__ __device__ constexpr uint32_t sortItemsFor(uint32_t digitBits) { return digitBits >= 9 ? 4u : 8u; }
__host__ __device__ constexpr uint32_t sortTileFor(uint32_t digitBits) { return kSortThreads * sortItemsFor(digitBits); }
constexpr uint32_t kSortMinTile = kSortThreads * 4u;

SortPlan makeSortPlan(uint32_t n, uint32_t bits, uint32_t maxDigitBits);
// Scratch layout inside one allocation.
struct SortScratch {
  uint32_t* hist;      // passes * bins
  uint32_t* counters;  // passes (tile counters)
  uint32_t* status;    // passes * tiles * bins
  uint2* tmp;          // n pairs (ping-pong), may be null for the engine
  size_t bytes;
};
size_t sortScratchBytes(const SortPlan& p, bool withTmp);
SortScratch carveSortScratch(const SortPlan& p, void* base, bool withTmp);

// Launch one onesweep pass.
cudaError_t launchOnesweepPass(const SortPlan& p, uint32_t pass, const uint2* in, uint2* out,
                               const SortScratch& s, uint32_t* errWord, cudaStream_t st);
// Histogram of all passes' digits (standalone sort only; the engine fuses it
// into the hash kernel).
cudaError_t launchSortHistogram(const SortPlan& p, const uint2* in, const SortScratch& s, uint32_t* errWord, cudaStream_t st);

// Thread-local error message.
void setLastError(const std::string& msg);
// A named range on a profiler's timeline (NVTX) for the duration of an entry
// point, as the reference timed its kernel calls (Core/DeviceInterface.cu:
// 389-456): the host-side span of the call, nested ranges included.  With no
// tool attached the push and pop cost a few nanoseconds.
struct TraceRange {
  explicit TraceRange(const char* name) { nvtxRangePushA(name); }
  ~TraceRange() { nvtxRangePop(); }
  TraceRange(const TraceRange&) = delete;
  TraceRange& operator=(const TraceRange&) = delete;
};

// A bad argument to entry point `fn`: records "fn: bad arguments" for
// brt_last_error and returns BRT_ERR_ARG.
inline int argError(const char* fn) {
  setLastError(std::string(fn) + ": bad arguments");
  return BRT_ERR_ARG;
}

}  // namespace brt

#define BRT_CUDA_TRY(expr)                                                              \
  do {                                                                                  \
    cudaError_t _e = (expr);                                                            \
    if (_e != cudaSuccess) {                                                            \
      ::brt::setLastError(std::string(#expr) + ": " + cudaGetErrorString(_e));          \
      return BRT_ERR_CUDA;                                                              \
    }                                                                                   \
  } while (0)
