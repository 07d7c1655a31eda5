// batch.hpp -- many independent instances of uneven sizes advanced together:
// each iteration is one captured graph in which the evaluator and the
// sampler are single launches over the children of every instance, and the
// per-instance steps (selection, incumbent, prune, pool rebuild, eviction)
// run as one thread block per instance in shared memory.
//
// Every instance follows the batched algorithm of the single-instance
// solver step for step (same selection order, salts, pool order, eviction
// and adaptive screen), so an instance's result does not depend on which
// other instances share the launches.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "../../include/cuminlp_gb300.h"
#include "kernels.cuh"

namespace cmn {

constexpr int kMiThreads = 1024;   // threads of a per-instance block
constexpr int kMiSortMax = 8192;   // largest pool a block holds (eight entries a thread)

struct BatchCfg {
  int n_max;        // variables per instance, at most
  int slots_max;    // program slots per instance, at most
  int log2C;        // B: children per parent = 2^B
  int max_slots;    // = B
  int precision;
  int sample_all;
  int relative;
  uint64_t S;
  uint64_t e_max;         // parents per instance per iteration
  uint64_t cap;           // pool capacity per instance
  uint64_t P;             // pool stride: cap + e_max << B
  uint64_t K;             // instance slots
  uint64_t child_stride;  // child slots per instance: e_max << B
  int64_t max_cycle;
  int64_t enumerate_cap;
  int g_max;                 // lanes per child at most (1: one lane per child)
  uint64_t eval_capacity;    // threads the bound launches keep resident
  uint64_t sample_capacity;  // threads the sample launch keeps resident
  int seg_max;               // lazy form: sum-chain segments per instance program, at most
  // instances whose program is a set of sum chains take the tile kernels
  // (batch_chain_kernels.cu), where their shared memory fits
  int tiles;                 // 1: it does
  int sms;
  int log_pts;               // points per warp of the tile samplers
  int lazy_chains;           // LazyShape
  int lazy_parts;
};

struct InstDesc {
  const Instr* prog64;
  const Instr* prog32;
  const int32_t* kinds;
  const double* root_lb;
  const double* root_ub;
  const int32_t* sched;  // lane schedules of the program (null: none)
  int32_t prog_len;
  int32_t n_vars;
  int32_t n_slots;
  int32_t active;
  int32_t g_max;        // lanes that may share one of its boxes
  int32_t pad_;
  uint64_t iter_limit;
  uint64_t batch_iter_limit;
  double tolerance;
  // lazy form: the FP32 point program, and the program's incremental
  // tables (Program::inc_*; inc_segments 0: the whole FP32 program bounds
  // each child)
  const Instr* prog32p;
  const int32_t* inc_seg;
  const int32_t* inc_off;
  const int32_t* inc_pcs;
  int32_t inc_segments;
  int32_t tile;  // 1: the instance takes the tile kernels
  ChainTab chain;
};

struct InstState {
  double gub;
  double glb;
  double dropped_lb_min;
  uint64_t pool_min_key;
  uint64_t pool_size;
  uint64_t n_parents;
  uint64_t salt_base;
  uint64_t expansions;
  uint64_t iterations;
  uint64_t remaining;
  uint64_t free_top;  // free store slots
  uint64_t kept;      // children the last iteration kept
  uint64_t viable;
  uint64_t dropped_min_key;
  uint32_t done;
  uint32_t converged;
  uint32_t have_best;
  uint32_t use_screen;
  Cand best;
  cmn_counters counters;
};

struct BatchBufs {
  InstDesc* desc;
  InstState* st;
  double* lo;  // [K][P][n_max]: the box store, a box contiguous
  double* hi;
  double* lb;  // [K][P] the pool in position order: lower bound,
  uint32_t* idx;         // [K][P] and store slot
  uint32_t* depth;       // [K][P] by store slot
  uint32_t* free_slots;  // [K][P] stack of free store slots (InstState::free_top)
  uint32_t* pslot;       // [K][e_max] store slots of the selected parents, in order
  uint32_t* klist;       // [K][child_stride] the kept children, in order,
  uint32_t* kslot;       // and their store slots
  double* plo;  // [K][n_max][e_max]
  double* phi;
  float* plo32;  // FP32 screen only: the same planes rounded outward
  float* phi32;
  uint32_t* pdepth;  // [K][e_max]
  ParentInfo* pinfo;
  SlotPlan* slots;  // [K][e_max][B]
  void* enum_scratch;  // [K][e_max][n_max]
  void* bis_scratch;
  uint64_t* heap_scratch;
  double* clb;  // [K][child_stride]
  uint8_t* cstate;
  double* cval;
  uint64_t* ce;
  uint32_t* list;  // certify list
  uint64_t* list_count;
  uint32_t* block_counts;
  uint32_t* block_offsets;
  uint64_t* child_base;  // [K + 2]: exclusive prefix of live children by `order` position, then the lane cap
  // the tile instances' work, as exclusive prefixes by `order` position
  // ([K + 1]): tiles of parents and of children for the constraints (2^live[1]
  // and 2^live[2] boxes each), tiles of 32 parents (lazy children), of 32
  // children (objective) and of 2^log_pts children (points)
  uint64_t* ptile;
  uint64_t* ctile;
  uint64_t* ltile;
  uint64_t* stile;
  uint64_t* qtile;
  uint64_t* live;           // [0] live children of all instances, [1], [2] as above,
                            // [3] most lanes any live instance can use per box
  uint64_t* stamps;         // [5] phase boundaries of the last iteration
  unsigned long long* sbest;  // [K] lb_key of the best point value known
  // [K]: the slots in the order the bound and sample launches walk their
  // children -- longest program first, so the launch's tail is short
  // programs (longest-processing-time-first balance)
  const uint32_t* order;
  double* best_point;  // [K][n_max]
  // lazy form
  double* plb;         // [K][e_max] the staged parents' certified FP64 lower bounds
  uint8_t* pfeas;      // [K][e_max] and their reference predicate
  float* inc_common;   // [K][seg_max][e_max] (lo, hi): chain sums without split variables
  float* inc_parts;    // [K][seg_max][2^B][e_max] (lo, hi): per slot part (incremental children)
  Best32* cbest;       // [K][child_stride] the FP32 screen's best sample per child
  // the verdict's warp runs: per `order` position the exclusive prefix of
  // its runs, then the total and the ticket the warps draw runs from
  uint64_t* vrun;      // [K + 2]
  uint8_t* vlg;        // [K] log2 of the lanes per parent of each position
};

#ifdef __CUDACC__
// Variable v of the staged parents of `slot`.
__device__ __forceinline__ size_t splane(const BatchCfg& c, uint64_t slot, int v)
{
  return ((size_t)slot * c.n_max + v) * c.e_max;
}

// Largest `order` position whose prefix does not exceed i.
__device__ __forceinline__ uint64_t position_of(const uint64_t* __restrict__ base, uint64_t K, uint64_t i)
{
  uint64_t lo = 0, hi = K;
  while (hi - lo > 1) {
    const uint64_t mid = (lo + hi) >> 1;
    if (__ldg(base + mid) <= i) lo = mid;
    else hi = mid;
  }
  return lo;
}
#endif

// The tile kernels of an iteration (batch_chain_kernels.cu): constraints of
// the staged parents (lazy form) or of the children, the lazy form's child
// bounds, the children's objectives, and the points.
struct BatchTileGrids {
  int constraints = 0, children = 0, lazy = 0, objective = 0, points = 0, picks = 0;
};
// Sets cfg's tile fields; 0 tiles when the kernels' shared memory is short.
void batch_tile_config(BatchCfg& cfg, int max_smem);
BatchTileGrids batch_tile_grids(const BatchCfg& cfg);
bool batch_tile_takes(const BatchCfg& cfg, const ChainTab& chain);
cudaError_t batch_tile_parents(const BatchCfg& cfg, const BatchBufs& b, const BatchTileGrids& g, cudaStream_t s);
cudaError_t batch_tile_lazy(const BatchCfg& cfg, const BatchBufs& b, const BatchTileGrids& g, cudaStream_t s);
cudaError_t batch_tile_children(const BatchCfg& cfg, const BatchBufs& b, const BatchTileGrids& g, cudaStream_t s);
cudaError_t batch_tile_points(const BatchCfg& cfg, const BatchBufs& b, const BatchTileGrids& g, cudaStream_t s);
cudaError_t set_batch_tile_attributes(int max_smem);

// Puts `slot`'s root box in its pool and resets its state.
cudaError_t batch_init_slot(const BatchCfg& cfg, const BatchBufs& b, uint64_t slot, double gub0, cudaStream_t s);
// Blocks of the grid-stride launches of an iteration.  `eval` serves the
// evaluators, the verdict and the samplers (their lane groups size
// themselves to it); the lazy form's FP32 sum and screen passes use fewer
// registers and take as many blocks as stay resident on the GPU.
struct BatchGrids {
  int eval = 1;
  int inc_common = 1;
  int inc_parts = 1;
  int screen = 1;
  BatchTileGrids tile;
};
BatchGrids batch_grids(const BatchCfg& cfg, int eval_grid);
// Enqueues one iteration over every active instance (capturable).
// The kernels write BatchBufs::stamps (ns) at the phase boundaries: start,
// after select + branch, after bound, after sample, after finish.
cudaError_t batch_iteration(const BatchCfg& cfg, const BatchBufs& b, const BatchGrids& grids, cudaStream_t s);
// The first m pool entries of `slot` in position order: boxes as (lower,
// upper) pairs (or null), lower bounds and depths.
cudaError_t batch_frontier(const BatchCfg& cfg, const BatchBufs& b, uint64_t slot, uint64_t m, double* boxes,
                           double* lower_bounds, uint32_t* depths, cudaStream_t s);
size_t batch_eval_smem(const BatchCfg& cfg, bool fp32);
size_t batch_sample_smem(const BatchCfg& cfg);
// resident blocks per SM of the bound (fp32: screen) and sample kernels
int batch_eval_occupancy(const BatchCfg& cfg, bool fp32);
int batch_sample_occupancy(const BatchCfg& cfg);
cudaError_t set_batch_kernel_attributes(int max_smem);

}  // namespace cmn
