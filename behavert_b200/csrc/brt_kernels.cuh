// brt_kernels.cuh -- argument blocks and launchers of the pipeline kernels.
#pragma once

#include "brt_internal.cuh"

namespace brt {

constexpr uint32_t kFusedThreads = 128;
constexpr uint32_t kFlockMaxThreads = 256;  // largest block of the single-pass flock kernel

struct HashArgs {
  const float4* pos;           // canonical slot order
  const uint32_t* id;          // agent id per canonical slot
  uint2* pairs;                // out, agent-id order: (key, slot)
  const FlockDev* flocks;
  const uint32_t* agentBase;   // nflocks + 1
  uint32_t nflocks, n;
  uint32_t passes, bins;
  uint32_t shift[4], mask[4];
  uint32_t* hist;              // passes * bins, accumulated with atomics
  uint32_t* cellStart;
  uint32_t* cellEnd;
  uint32_t cellWords4;         // cell words / 4 (arrays padded to 4)
  uint32_t* status;            // sort look-back state to clear
  uint32_t statusWords;
  uint32_t* counters;          // sort tile counters to clear
  uint32_t* stepCounter;       // random-stream step counter, incremented once per step
};

struct ReorderArgs {
  const uint2* pairs;          // sorted (key, previous slot)
  const float4* posA; const float4* fwdA; const float4* accA;
  const float* featA; const uint32_t* idA;
  float4* posS; float4* fwdS; float4* accS; float* featS; uint32_t* idS;
  uint32_t* prevOut;           // source slot per sorted slot (optional, adjoint tape)
  uint32_t fs4;                // feature float4s per agent
  uint32_t* cellStart; uint32_t* cellEnd;
  uint32_t* hist; uint32_t histWords;
  uint32_t n, numCells;
  uint32_t* errWord;
  // the order by counting (reorderKernel<true>): the cells' members, whose
  // ranks it takes, and the sorted pairs it writes; null with the radix sort
  const uint4* members;
  uint2* pairsOut;
  // engines whose flocks differ in featuresCount: the sorted features with only
  // each flock's own columns, the others zero (null: all flocks own all columns)
  float* featOwn;
  // cell-cull gate of scan variants 0 and 1 (null: not computed).  Words
  // [0] and [1] are the launch's accumulator and block ticket, both back at
  // zero when the launch ends; [2] is set to nonzero when a sorted position
  // is NaN or outside [0, L] on some axis of its flock's world.
  uint32_t* cullWords;
  const FlockDev* flocks; const uint32_t* agentBase; uint32_t nflocks;
};

struct FusedArgs {
  const float4* posS; const float4* fwdS; const float4* accS;
  const float* featS; const uint32_t* idS;
  float4* posA; float4* fwdA; float4* accA; float* featA; uint32_t* idA;
  float4* statsById;
  bool clus;                   // some flock has clustering steering
  float4* steerOut;            // optional: the steering force of every sorted slot (adjoint tape)
  const uint32_t* cellStart; const uint32_t* cellEnd;
  const FlockDev* flocks; const uint32_t* agentBase;
  const float4* obstacles;
  const uint2* obsMask;          // per-cell obstacle field (global cell index) or null
  uint32_t* lists;             // optional, stride listStride
  uint32_t listStride;
  uint32_t nflocks, n, Mmax, Fs;
  uint32_t warpAgents;         // agents a warp of a cooperative scan takes (agentOfLane)
  uint32_t smCount;            // SMs of the device, for the host's rules
  float dt;
  int scanVariant;             // 0: pipelined x4 + cell culling, 1: x2 + culling, 2: x4, 3: flat loop,
                               // 4: warp-cooperative, 5: warp-cooperative with windows,
                               // 6: staged tiles (tileFlockKernel), 7: warp-cooperative with
                               // bounding-box culling
  const uint32_t* stepCounter; // random-stream step of the Schooling move
  const uint32_t* cullGate;    // scan variants 0 and 1: cells are culled only when
                               // this word is zero (null: never culled)
  // scan variant 6: the (flock, row segment) tiles and the work-queue counter
  const uint4* tiles;          // x flock, y row y | z << 16, z first x | cells << 16
  uint32_t numTiles;
  uint32_t* tileCounter;       // zeroed before each launch
  uint32_t tileBlocks;         // persistent blocks of the launch
};
// Home cells per tile (one row segment) and staged candidates per tile.
constexpr uint32_t kTileMaxCells = 32;
constexpr uint32_t kTileThreads = 128;

struct StageArgs {
  const float4* posS; const float4* fwdS; const float4* accS;
  const float* featS; const uint32_t* idS;
  float4* posA; float4* fwdA; float4* accA; float* featA; uint32_t* idA;
  float4* statsById;
  float4* steer;
  float4* fwdW;                  // the sorted forwards again, written by the avoid-neighbours stage
  float avoidBase[3];            // move-away stage: the point to flee
  float avoidBaseParams[3];      //   (steering weight, acceleration factor, radius)
  const uint32_t* cellStart; const uint32_t* cellEnd;
  const FlockDev* flocks; const uint32_t* agentBase;
  const float4* obstacles;
  const uint2* obsMask;          // per-cell obstacle field (global cell index) or null
  uint32_t* lists;
  uint32_t listStride;
  uint32_t nflocks, n, Fs;
  uint32_t warpAgents;         // agents a warp of a cooperative scan takes (agentOfLane)
  const uint32_t* stepCounter;
};

// The order by counting (brt_order.cu).  reorderKernel ranks the members of a
// cell by comparing their ids; those of a cell of more than kRankLimit placeKernel
// sorts instead.  us of a warm order of 1,000,000 agents ranked / sorted (and by the
// radix sort): 500 a cell 115 / 132 (63), 700: 145 / 105 (64), 1,000: 188 / 101 (65),
// 2,000: 324 / 131 (62), 4,000: 1,724 / 158 (60).
constexpr uint32_t kRankLimit = 512;
// Of those, the cells of more than giantLimit, at most kGiants, are sorted together
// by all blocks; a block each sorts the others.  So no block is left with more than
// 1 / 256 of the agents: 1,000,000 in one cell 95 us (radix sort 43; with one block
// for every cell above 4,096 it was 14,300), in 27 cells 103 (46; 14,600); 100,000
// in one cell 38 (22; 1,380).
constexpr uint32_t kGiants = 256;
__host__ __device__ constexpr uint32_t giantLimit(uint32_t n) { return n / kGiants > kRankLimit ? n / kGiants : kRankLimit; }
// Agents a tile of that takes.  us of a warm order with 1,024 / 2,048 / 4,096:
// 1,000,000 agents in one cell 99 / 103 / 109, in 250 cells (half of them giants)
// 264 / 166 / 221; 100,000 in 27 cells 40 / 43 / 57.
constexpr uint32_t kGiantTile = 2048;
__host__ __device__ constexpr uint32_t bigCellCap(uint32_t n) { return n / kRankLimit + 1; }
// scan tiles claimed, place blocks done, crowded cells of a block each, giant
// cells, work items claimed
constexpr uint32_t kOrderWordTile = 0, kOrderWordDone = 1, kOrderWordBig = 2, kOrderWordGiant = 3, kOrderWordItem = 4;
constexpr uint32_t kOrderWords = 8;
struct OrderArgs {
  const float4* pos;             // canonical positions
  const uint32_t* id;            // agent id per canonical slot
  const FlockDev* flocks; const uint32_t* agentBase;
  uint32_t nflocks, n, numCells;
  uint2* cellPlace;              // [n] (cell, place among the cell's agents) per canonical slot
  uint32_t* count;               // [numCells, padded] zero between steps
  uint32_t* cellStart; uint32_t* cellEnd;
  uint4* members;                // [n] by cell: (id, canonical slot, cell's first position, cell)
  uint2* scratch[2];             // [n] each: the pair buffers, for crowded cells
  uint32_t* giantStatus;         // [tiles of kGiantTile agents x kGiants] look-back state, in a staging buffer
  uint32_t* tileStatus;          // [cell tiles] look-back state of the cell scan
  uint32_t* giantCells;          // [kGiants]
  uint32_t* bigCells;            // [bigCellCap(n)]
  uint32_t* words;               // [kOrderWords]
  uint32_t* stepCounter;         // random-stream step, advanced once per step
  uint32_t* errWord;
  LookbackWait wait;             // bound of the cell scan's look-back
};
uint32_t orderCellTiles(uint32_t numCells);
cudaError_t launchOrderCount(const OrderArgs& A, cudaStream_t st);
cudaError_t launchOrderPlace(const OrderArgs& A, cudaStream_t st);

// Agents a warp of a warp-cooperative scan takes: 32, or fewer when that many
// warps would leave the GPU part empty.  A warp goes through its home cells'
// runs one after the other (about 5 us a run of 4 agents), so a launch that
// does not fill the GPU lasts as long as one warp's chain; 4 agents are about
// one run.  With fewer agents a warp the runs are cut into more pieces and the
// list walk has fewer lanes, so the line is at half a wave of resident warps
// (flockWarpAgents: a full wave where the launch runs alone): a launch alone
// would gain a little more from a full wave, several engines at once lose by it.
// Measured, us a step alone with 32 / 16 / 8 / 4 agents a warp (maxNeighbors 16,
// density 1/16, 148 SMs of 32 resident warps): 4,096 agents 59.2 / 48.2 / 42.7 /
// 39.2; 16,384: 64.0 / 53.0 / 47.5 / 46.7; 32,768: 68.0 / 56.6 / 53.2 / 65.5;
// 65,536: 73.1 / 65.0 / 76.5 / 97.2; 100,003: 83.3 / 90.0 / 100.4 / 131.8.  Three
// engines of 73,029 schooling agents in turn, us a step: 36.5 with 32, 42.0 with 16.
inline uint32_t warpAgentsFor(uint32_t n, uint32_t residentWarps) {
  for (uint32_t a = 4; a < 32; a *= 2)
    if ((n + a - 1) / a <= residentWarps) return a;
  return 32;
}
int flockKnnScan(uint32_t block, uint32_t Mmax, int regs);
uint32_t flockWarpAgents(const FusedArgs& A, uint32_t block, int phase2, int regs);
uint32_t fusedWarpAgents(uint32_t n, uint32_t Mmax, uint32_t smCount);
uint32_t listsWarpAgents(uint32_t n, uint32_t Mmax, uint32_t smCount);
uint32_t schoolWarpAgents(uint32_t n, uint32_t Mmax, uint32_t smCount);


// Reverse of one taped step (brt_adjoint.cu).
constexpr uint32_t kAdjointThreads = 128;
struct AdjointStepArgs {
  uint32_t smCount;                                              // of the device, for the host's rule
  const float4* posS; const float4* fwdS; const float4* accS;   // the step's sorted input state
  const float4* steerS;                                          // and the steering force of its forward
  const uint32_t* lists; uint32_t listStride;                    // its neighbour lists (sorted slots)
  const uint32_t* prev;                                          // canonical slot of each sorted slot
  const uint32_t* idS;                                           // agent id per sorted slot
  const FlockDev* flocks; const uint32_t* agentBase; const float4* obstacles;
  const uint2* obsMask;
  uint32_t nflocks, n;
  float dt;
  const float4* gOutP; const float4* gOutF; const float4* gOutA; // output adjoint by sorted slot
  float4* gInP; float4* gInF; float4* gInA;                      // input adjoint by canonical slot
  // Emit -> gather hand-over of one step (sorted slots of this step):
  float4* contrib;      // 2 per list entry e = i * entryStride + k, for in-list overflow only: the
                        // position adjoint (xyz) and forward adjoint (w, then xy) agent i sends
                        // the agent it lists at k
  float4* selfP;        // per slot: the agent's own position adjoint terms
  float4* selfF;        // per slot: the agent's own forward adjoint terms (w: speed)
  // In-lists (the transposed neighbour list of the step): the contribution
  // of entry e = i * entryStride + k (agent i lists j at position k) goes to
  // inbox[2 * (j * inCap + q)] (two float4) at q = atomicAdd(&inCount[j], 1);
  // entries beyond inCap go to contrib[2 * e] and a linked overflow list
  // (ovHead[j], ovNext[e]).  The gather resets inCount and ovHead for the
  // next-earlier step.
  uint32_t* inCount; float4* inbox; uint32_t inCap;
  uint32_t* ovHead; uint32_t* ovNext;
  uint32_t entryStride; // list positions per slot in the entry code (maxNeighbors, <= 32)
  double* accW;         // per agent id: the weight adjoint summed over the steps (3 doubles)
  uint32_t* exportLists;                                         // optional, by agent id
  uint32_t* exportFlags;                                         // optional, 4 words by agent id
  float4* exportState;                                           // optional: pos, fwd, acc by agent id
};
constexpr uint32_t kNoEntry = 0xFFFFFFFFu;
// Per-flock FP64 sums of per-item values (the weight adjoint, the loss), in
// a fixed order: kReduceParts blocks per flock, each over a fixed part of the
// flock's items, then the parts in order.
constexpr uint32_t kReduceParts = 32;
struct FlockReduceArgs {
  const double* vals; uint32_t width;   // width (1..3) doubles per item
  const uint32_t* agentBase;            // items of flock f: [agentBase[f], agentBase[f+1])
  uint32_t nflocks;
  double* partial;                      // nflocks * kReduceParts * width scratch
  double* out;                          // nflocks * width, written
};
struct LossArgs {
  const float4* posA; const uint32_t* idA;    // final state, canonical order
  const float4* target;                       // by agent id
  const FlockDev* flocks; const uint32_t* agentBase;
  uint32_t nflocks, n;
  double* lossTerm;                           // per canonical slot (reduced per flock afterwards)
  float4* gT;                                 // unscaled terminal position adjoint, canonical order
};
struct SeedArgs {
  const float4* gT; const float* scale;       // scale per flock (device) or null for 1
  const float4* extraP; const float4* extraF; const float4* extraA;  // optional, by agent id
  const uint32_t* idA;
  const uint32_t* agentBase;
  uint32_t nflocks, n;
  float4* gP; float4* gF; float4* gA;
};
struct OutArgs {
  const float4* gP; const float4* gF; const float4* gA;
  const uint32_t* id0; const float4* fwd0;    // initial canonical order
  uint32_t n;
  float4* outP; float4* outF; float4* outA; float4* outV;  // by agent id, each optional
};
cudaError_t launchAdjointStep(const AdjointStepArgs& A, cudaStream_t st);
cudaError_t launchFlockReduce(const FlockReduceArgs& A, cudaStream_t st);
cudaError_t launchLoss(const LossArgs& A, cudaStream_t st);
cudaError_t launchAdjointSeed(const SeedArgs& A, cudaStream_t st);
cudaError_t launchAdjointOut(const OutArgs& A, cudaStream_t st);

cudaError_t launchHash(const HashArgs& A, uint32_t maxBlocks, cudaStream_t st);
// Canonical features of sorted slot i beyond its flock's own columns, from its sorted row.
cudaError_t launchCarryColumns(const float* featS, float* featA, uint32_t Fs, const FlockDev* flocks, const uint32_t* agentBase,
                               uint32_t nflocks, uint32_t n, cudaStream_t st);
cudaError_t launchReorder(const ReorderArgs& A, cudaStream_t st);
cudaError_t launchFused(const FusedArgs& A, bool knn, cudaStream_t st);
cudaError_t launchFlock(const FusedArgs& A, int phase2, uint32_t block, int regs, cudaStream_t st);
uint32_t tileFlockBlocks(uint32_t Mmax, uint32_t Fs, int smCount);
cudaError_t launchLists(const StageArgs& A, bool knn, cudaStream_t st);
cudaError_t launchSteerStage(const StageArgs& A, int which, cudaStream_t st);
cudaError_t launchIntegrateStage(const StageArgs& A, float dt, cudaStream_t st);
// Schooling (brt_school.cu): fused step, and stage which = 0 repulsion,
// 1 attraction/orientation, 2 move, 3 animateSchool.
cudaError_t launchSchool(const FusedArgs& A, cudaStream_t st);
cudaError_t launchSchoolStage(const StageArgs& A, int which, cudaStream_t st);
cudaError_t configureSchoolKernels(uint32_t Mmax);
// BehaviorClustering analytics (brt_cluster.cu): which = 0 reset labels,
// 1 one propagation sweep, 2 hit rate; in / out are the membership buffers.
struct ClusterArgs {
  const float4* posS; const uint32_t* idS;
  const uint32_t* lists; uint32_t listStride;
  const FlockDev* flocks; const uint32_t* agentBase;
  uint32_t nflocks, n;
  float radius;
  const float4* in; float4* out;
};
cudaError_t launchCluster(const ClusterArgs& A, int which, cudaStream_t st);
// State between agent-id order and the canonical slot order; a null source
// leaves its array out.
struct StateIoArgs {
  const float4* src[3]; float4* dst[3];  // positions, forwards, smoothed accelerations
  const float* featSrc; float* featDst;
  uint32_t F, Fs;                        // floats an agent: outside, and in the canonical array
  const uint32_t* id;                    // agent id per canonical slot
  uint32_t n;
};
cudaError_t launchStateIo(const StateIoArgs& A, bool gather, cudaStream_t st);
cudaError_t configureFusedKernels(uint32_t Mmax);
cudaError_t configureFlockKernels(uint32_t Mmax);
cudaError_t launchHashPairsOut(const uint2* pairs, const uint32_t* idS, uint32_t* keys, uint32_t* ids, uint32_t n, cudaStream_t st);
// dst[i] = src[index[i * stride]] and dst[index[i]] = src[i] for arrays of
// `words` 32-bit words per agent.
cudaError_t launchGatherWords(const uint32_t* src, const uint32_t* index, uint32_t stride, uint32_t* dst, uint32_t words,
                              uint32_t n, cudaStream_t st);
cudaError_t launchScatterWords(const uint32_t* src, const uint32_t* index, uint32_t* dst, uint32_t words, uint32_t n,
                               cudaStream_t st);

uint32_t sortPassMask(const SortPlan& p, uint32_t pass);

}  // namespace brt
