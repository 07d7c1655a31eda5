// chain_points.cu -- the sampler and the lazy form's FP32 sample screen over
// one instance whose program is a set of sum chains (point_tiles.cuh).
#include <cfloat>
#include <cstdint>

#include "launch.hpp"
#include "point_tiles.cuh"

namespace cmn {

// Point sampling and exact points (sample_children_kernel's results): every
// point is drawn in FP64 and its constraints are summed in FP32; only a point
// they do not exclude, and whose FP32 objective does not prove it worse than
// the best point of this block (or, in the solver, than the incumbent), is
// evaluated in FP64.  The best candidate is the same: what is left out is
// infeasible or strictly worse than a candidate that was evaluated.
//
// A warp takes 2^log_pts points at a time, then evaluates the points left one
// by one with all its lanes, the FP32-best first, so that one FP64 evaluation
// usually rules out the others.  Taken
// where every chain has a filter and the boxes are within its range
// (ChainTab::points): elsewhere too many points would be left.
// kChunks: the points are the lazy form's picks, one per chunk of children.
template <bool kChunks>
__global__ void __launch_bounds__(kPointThreads) chain_sample_kernel(const SampleArgs a, int log_pts)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned long long best_s;  // lb_key of the block's best value so far
  __shared__ uint8_t list_s[kPointThreads];
  const int pts = 1 << log_pts;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, W = blockDim.x >> 5;
  const int n = a.n_vars;
  double* x64 = reinterpret_cast<double*>(smem_raw) + (size_t)wid * n;
  float* x32 = reinterpret_cast<float*>(smem_raw + (size_t)W * n * 8 + wid * point_bytes(n, log_pts));
  uint8_t* list = list_s + wid * 32;
  if (a.done != nullptr && *a.done) {
    if (threadIdx.x == 0) a.block_best[blockIdx.x] = Cand{INFINITY, 0xffffffffu, 0, ~0ULL};
    return;
  }
  stamp_first(a.t_first);
  const uint64_t children = a.n_children_dev ? *a.n_children_dev : a.n_children;
  const uint64_t per = a.exact ? 1 : a.S;
  const uint64_t total = kChunks ? (children + (1ULL << kChunkLog2) - 1) >> kChunkLog2 : children * per;
  const uint64_t salt_base = a.salt_base_dev ? *a.salt_base_dev : 0;
  const double gub = a.gub ? *a.gub : DBL_MAX;
  const bool solver = a.state != nullptr;
  // a solver's candidate must be below the incumbent to count
  if (threadIdx.x == 0) best_s = lb_key(solver ? gub : INFINITY);
  __syncthreads();
  Cand best = {INFINITY, 0xffffffffu, 0, ~0ULL};
  unsigned long long rejected = 0;
  const uint64_t warps = (uint64_t)gridDim.x * W;
  for (uint64_t w0 = (uint64_t)blockIdx.x * W + wid; w0 << log_pts < total; w0 += warps) {
    // lane < pts: its point
    const uint64_t item = (w0 << log_pts) + lane;
    PointOf p = {};
    bool cand = lane < pts && item < total;
    if (kChunks) {
      cand = cand && chunk_point(a, item, children, salt_base, p);
    } else if (cand) {
      const uint64_t g = item / per;
      p.i = item - g * per;
      cand = point_child(a, g, salt_base, p) && (!p.fathom || p.i == 0);
    }
    sample_tile(a, x64, x32, list, log_pts, p, cand, &best_s, gub, rejected, [&](const PointOf& o, double value) {
      const Cand c = {value, (uint32_t)o.k, 0, o.r * (o.fathom ? 1 : a.S) + o.i};
      if (cand_less(c, best)) best = c;
    });
  }
  best = block_min_cand(best);
  if (threadIdx.x == 0) a.block_best[blockIdx.x] = best;
  if (a.rejected != nullptr) {
    for (int off = 16; off > 0; off >>= 1) rejected += __shfl_down_sync(0xffffffffu, rejected, off);
    if (lane == 0 && rejected) atomicAdd(a.rejected, rejected);
  }
}

__global__ void __launch_bounds__(kPointThreads) chain_screen_kernel(const SampleArgs a, int log_pts)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint8_t list_s[kPointThreads];
  const int wid = threadIdx.x >> 5, W = blockDim.x >> 5;
  float* x = reinterpret_cast<float*>(smem_raw + wid * point_bytes(a.n_vars + 1, log_pts));
  if (a.done != nullptr && *a.done) return;
  stamp_first(a.t_first);
  const uint64_t total = a.n_children_dev ? *a.n_children_dev : a.n_children;
  const uint64_t salt_base = a.salt_base_dev ? *a.salt_base_dev : 0;
  for (uint64_t w0 = (uint64_t)blockIdx.x * W + wid; w0 << log_pts < total; w0 += (uint64_t)gridDim.x * W)
    screen_tile(a, x, list_s + wid * 32, log_pts, w0, total, salt_base);
}

// ---- launchers ----
static size_t sample_smem(int n, int log_pts) { return (size_t)(kPointThreads / 32) * ((size_t)n * 8 + point_bytes(n, log_pts)); }
static size_t screen_smem(int n, int log_pts) { return (size_t)(kPointThreads / 32) * point_bytes(n + 1, log_pts); }

bool chain_sample_fits(const SampleArgs& a)
{
  return a.chain.points && a.sched != nullptr &&
         sample_smem(a.n_vars, 0) + 2048 <= (size_t)max_dynamic_smem();
}

cudaError_t launch_chain_sample(const SampleArgs& a, int grid, cudaStream_t s)
{
  int lp = log_points(a.n_vars);
  if (a.n_children_dev == nullptr) {  // few points: more lanes on each
    const uint64_t warps = (uint64_t)grid * (kPointThreads / 32), points = a.n_children * a.S;
    while (lp > 0 && (points >> lp) < warps) --lp;
  }
  if (a.cbest != nullptr) chain_sample_kernel<true><<<grid, kPointThreads, sample_smem(a.n_vars, lp), s>>>(a, lp);
  else chain_sample_kernel<false><<<grid, kPointThreads, sample_smem(a.n_vars, lp), s>>>(a, lp);
  return cudaGetLastError();
}

bool chain_screen_fits(const SampleArgs& a)
{
  return a.chain.term_pt != nullptr && screen_smem(a.n_vars, 0) + 1024 <= (size_t)max_dynamic_smem();
}

cudaError_t launch_chain_screen(const SampleArgs& a, uint64_t max_children, cudaStream_t s)
{
  const int lp = log_points(a.n_vars + 1);
  const size_t smem = screen_smem(a.n_vars, lp);
  int occ = 1;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, chain_screen_kernel, kPointThreads, smem);
  if (e != cudaSuccess) return e;
  const uint64_t need = ((max_children >> lp) + kPointThreads / 32) / (kPointThreads / 32);
  const uint64_t room = (uint64_t)sm_count() * (uint64_t)(occ > 0 ? occ : 1);
  chain_screen_kernel<<<(unsigned)(need < room ? need : room), kPointThreads, smem, s>>>(a, lp);
  return cudaGetLastError();
}

cudaError_t set_chain_points_attributes(int max_smem)
{
  cudaError_t e = allow_dynamic_smem(chain_sample_kernel<false>, max_smem);
  if (e == cudaSuccess) e = allow_dynamic_smem(chain_sample_kernel<true>, max_smem);
  return e == cudaSuccess ? allow_dynamic_smem(chain_screen_kernel, max_smem) : e;
}

}  // namespace cmn
