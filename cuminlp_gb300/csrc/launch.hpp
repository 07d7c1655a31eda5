// launch.hpp -- host-side launch wrappers of the device kernels.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "kernels.cuh"

namespace cmn {

constexpr int kEvalThreads = 128;
// resident blocks per SM the single-instance bound kernels are compiled
// for (registers): 5 measured ahead of 4 and 6 on the n=32 and n=4
// workloads, with a little spilling
#ifndef CMN_EVAL_MIN_BLOCKS
#define CMN_EVAL_MIN_BLOCKS 5
#endif

// interval kernels: program slots plus `max_slots` split variables per thread
size_t eval_smem_bytes(int n_slots, int max_slots, bool fp32, int threads);
// sampler: one point column (variables + slots, FP64) per 2^lg_min threads
size_t sample_smem_bytes(int n_vars, int n_slots, int threads, int lg_min);
// Point columns of a block stay within this many bytes: lanes share a
// column (2^lg_min of them) until they do, so the sampler's residency does
// not fall with the number of variables.  Programs with shared slots have
// no lane schedule and keep one column per thread.
constexpr size_t kSampleColumnBytes = 32 * 1024;
int sample_lg_min(int n_vars, int n_slots, bool has_sched, int threads);
size_t sample_screen_smem_bytes(int n_vars, int n_slots, int threads, int lg_min);
// the lazy form's FP32 sample screen: one point column (FP32) per 2^lg_min lanes
int sample_screen_lg_min(int n_vars, int n_slots, bool has_sched, int threads);

// mode 0: role / raw boxes; 1: solver FP64; 2: solver FP32 screen (fp32
// must be true); 3: solver FP64 certify over EvalArgs::list; 4: aggregate
// bounder (FP64, per-child fold into EvalArgs::agg_keys); 5: solver lazy
// form, FP32 children bounded by the parents' certified bounds (fp32 true);
// 6: the lazy form's FP64 verdict of the staged parents (mode 0's outputs,
// each term's coefficient and chain add fused into __fma_rd / __fma_ru)
cudaError_t launch_eval(const EvalArgs& a, int mode, bool fp32, int grid, int threads, cudaStream_t s);
// The FP64 modes over a program of sum chains (EvalArgs::chain):
// chain_kernels.cu.  chain_fits: whether the launch can take that path;
// chain_pays: whether it is the faster one.
bool chain_fits(const EvalArgs& a);
bool chain_pays(const EvalArgs& a, int mode);
cudaError_t launch_chain(const EvalArgs& a, int mode, cudaStream_t s);
cudaError_t set_chain_kernel_attributes(int max_smem);
// mode 0 over few boxes of a program in levels (level_kernels.cu)
bool level_fits(const EvalArgs& a, bool fp32);
cudaError_t launch_level(const EvalArgs& a, bool fp32, cudaStream_t s);
cudaError_t set_level_kernel_attributes(int max_smem);
// FP32 modes 0 (boxes) and 2 (screen) over such a program, and the lazy
// form's child bounds (chain32_kernels.cu)
bool chain32_fits(const EvalArgs& a, int mode);
bool chain32_pays(const EvalArgs& a, int mode);
cudaError_t launch_chain32(const EvalArgs& a, int mode, cudaStream_t s);
bool lazy_children_fits(const ChainTab& t, int n_vars, int max_slots, int log2C);
cudaError_t launch_lazy_children(const EvalArgs& a, uint64_t max_parents, cudaStream_t s);
cudaError_t set_chain32_kernel_attributes(int max_smem);
// the sampler over such a program
bool chain_sample_fits(const SampleArgs& a);
cudaError_t launch_chain_sample(const SampleArgs& a, int grid, cudaStream_t s);
// the lazy form's FP32 sample screen over such a program
bool chain_screen_fits(const SampleArgs& a);
cudaError_t launch_chain_screen(const SampleArgs& a, uint64_t max_children, cudaStream_t s);
cudaError_t set_chain_points_attributes(int max_smem);
cudaError_t launch_sample(const SampleArgs& a, int grid, int threads, cudaStream_t s);
// the lazy form's incremental FP32 children: the common chain sums per
// (segment, parent), then every child (EvalArgs::inc_* set, prog = FP32)
cudaError_t launch_inc(const EvalArgs& a, int grid, int threads, cudaStream_t s);
// shared memory of the incremental child pass per block
size_t inc_child_smem_bytes(int max_slots, int threads);
// the lazy form's FP32 sample screen (SampleArgs::cbest out, prog = the
// FP32 point program)
cudaError_t launch_sample_screen(const SampleArgs& a, int grid, int threads, cudaStream_t s);
cudaError_t launch_candidate(const Cand* block_best, int n, Cand* out, const WitnessArgs& w, const Incumbent& inc,
                             cudaStream_t s);

// Largest dynamic shared memory a block may use on this device.
int max_dynamic_smem();

// Kernel attributes are set once per device, before any launch, so that
// launches stay legal inside stream capture.  The dynamic allowance is the
// opt-in maximum less the kernel's own static shared memory.
template <typename K>
cudaError_t allow_dynamic_smem(K kernel, int max_smem)
{
  cudaFuncAttributes fa;
  cudaError_t e = cudaFuncGetAttributes(&fa, kernel);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem - (int)fa.sharedSizeBytes);
}

// Resident blocks per SM of the sampler at this shared-memory size.
int sample_kernel_occupancy(size_t smem, int threads);
int sample_screen_occupancy(size_t smem, int threads);
int sm_count();

// Blocks of a launch whose kernel strides over `blocks` blocks' work: as many
// as are resident at once, no more than that.
template <typename K>
uint64_t resident_blocks(uint64_t blocks, K kernel, int threads, size_t smem)
{
  int occ = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, threads, smem) != cudaSuccess) (void)cudaGetLastError();
  const uint64_t room = (uint64_t)sm_count() * (uint64_t)(occ < 1 ? 1 : occ);
  return blocks < 1 ? 1 : blocks < room ? blocks : room;
}

}  // namespace cmn
