// handles.hpp -- definitions shared by the C ABI translation units.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "../../include/cuminlp_gb300.h"
#include "program.hpp"

// A compiled problem resident on one device.
struct cmn_problem {
  cmn::HostProblem host;
  cmn::Program prog;
  int device = 0;
  cmn::Instr* d_prog64 = nullptr;
  cmn::Instr* d_prog32 = nullptr;
  cmn::Instr* d_prog32p = nullptr;  // FP32 point program (the lazy form's sample screen)
  int32_t* d_kinds = nullptr;
  double* d_root_lb = nullptr;
  double* d_root_ub = nullptr;
  int32_t* d_sched = nullptr;  // lane schedules (Program::sched), null when none
  int32_t* d_inc_seg = nullptr;  // incremental child tables (Program::inc_*), null when none
  int32_t* d_inc_off = nullptr;
  int32_t* d_inc_pcs = nullptr;
  cmn::ChainSeg* d_chain_seg = nullptr;  // sum chains (Program::chain_*), null when none
  cmn::ChainTerm* d_chain_term = nullptr;
  cmn::ChainTerm32* d_chain_term32 = nullptr;
  cmn::ChainTerm32* d_chain_var32 = nullptr;
  int32_t* d_chain_var_off = nullptr;
  cmn::ChainTerm* d_chain_term_pt = nullptr;
  cmn::Instr* d_prog64l = nullptr;  // the program in levels (Program::level_*), null when none
  cmn::Instr* d_prog32l = nullptr;
  int32_t* d_level_off = nullptr;
  int32_t* d_level_run = nullptr;
  // one allocation holds every table above
  void* d_tables = nullptr;
  // host-buffer calls of cmn_eval_boxes stage through this, up to
  // kEvalWorkspace bytes; a second call at the same time takes its own
  mutable std::mutex ws_mu;
  mutable unsigned char* d_ws = nullptr;
  mutable size_t ws_bytes = 0;
  // cmn_autotune's choice per precision (0 FP64, 1 FP32): blocks per SM
  // and lanes per box cap; 0 = not tuned
  int tuned_bps[2] = {0, 0};
  int tuned_lanes[2] = {0, 0};

  cmn::ChainTab chain() const
  {
    cmn::ChainTab t{};
    if (!d_chain_seg) return t;
    t.seg = d_chain_seg;
    t.term = d_chain_term;
    t.n_seg = (int32_t)prog.chain_seg.size();
    t.pure_objective = prog.chain_seg[0].kind == cmn::kChainObjective ? 1 : 0;
    t.points = prog.chain_points ? 1 : 0;
    t.term32 = d_chain_term32;
    t.var32 = d_chain_var32;
    t.var_off = d_chain_var_off;
    t.term_pt = d_chain_term_pt;
    t.n_vars = (int32_t)host.n_vars();
    t.products = prog.chain_products;
    // no more warps than the terms over the longest chain, at most eight
    int64_t most = 1, all = 0;
    for (const cmn::ChainSeg& s : prog.chain_seg) {
      const int64_t len = s.pc1 - s.pc0;
      all += len;
      if (len > most) most = len;
      if (s.kind == cmn::kChainLe) {
        t.constraints += 1;
        t.constraint_terms += (int32_t)len;
      } else if (s.kind == cmn::kChainGeneral) {
        t.general += 1;
        t.general_terms += (int32_t)len;
      }
    }
    const int64_t w = (all + most - 1) / most;
    t.warps32 = (int32_t)(w < 1 ? 1 : w > 8 ? 8 : w);
    return t;
  }

  cmn::LevelTab levels() const
  {
    cmn::LevelTab t{};
    if (!d_level_off) return t;
    t.prog64 = d_prog64l;
    t.prog32 = d_prog32l;
    t.off = d_level_off;
    t.run = d_level_run;
    t.levels = (int32_t)(prog.level_off.size() - 1) / cmn::kLevelWarps;
    t.slots = prog.level_slots;
    return t;
  }

  ~cmn_problem();
};

namespace cmn {

constexpr size_t kEvalWorkspace = 64u << 20;

// How `planes` planes of n_boxes doubles, `stride` apart, go to the device:
// packed ones in one copy (33 boxes of two variables: 56 us a call, 73 by a
// pitched copy), others in one pitched copy, or plane by plane where the
// pitch is above the device's largest (documented as 2^31 - 1 bytes).
enum class PlaneCopy { kPacked, kPitched, kEach };
inline PlaneCopy plane_copy(uint64_t planes, uint64_t n_boxes, uint64_t stride, uint64_t max_pitch)
{
  if (stride == n_boxes || planes == 1) return PlaneCopy::kPacked;
  return stride > max_pitch / sizeof(double) ? PlaneCopy::kEach : PlaneCopy::kPitched;
}

// Collects arrays and gives them places in one device allocation: a solver
// has some forty, and each cudaMalloc / cudaFree of its own took 30-80 us.
class Slab {
 public:
  template <typename T>
  void add(T** ptr, size_t n)
  {
    const size_t bytes = (n > 0 ? n : 1) * sizeof(T);
    parts_.push_back({reinterpret_cast<void**>(ptr), total_});
    total_ += (bytes + 255) & ~(size_t)255;
  }
  size_t bytes() const { return total_; }
  cudaError_t alloc(void** base)
  {
    *base = nullptr;
    cudaError_t e = cudaMalloc(base, total_ > 0 ? total_ : 256);
    if (e == cudaSuccess)
      for (auto& p : parts_) *p.first = static_cast<unsigned char*>(*base) + p.second;
    return e;
  }

 private:
  std::vector<std::pair<void**, size_t>> parts_;
  size_t total_ = 0;
};

// Records `msg` as this thread's cmn_last_error() and returns `st`.
cmn_status set_error(cmn_status st, const std::string& msg);

// Sets the kernels' dynamic shared-memory allowance once per device.
cudaError_t ensure_kernel_attributes();

}  // namespace cmn
