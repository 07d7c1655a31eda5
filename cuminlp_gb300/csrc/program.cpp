// program.cpp -- validation and the DAG -> fused program compiler.
#include "program.hpp"

#include <algorithm>
#include <array>
#include <cfloat>
#include <cmath>
#include <cstring>

namespace cmn {

float d2f_rd(double x)
{
  if (std::isnan(x)) return (float)x;
  float f = (float)x;
  if (std::isinf(f) && !std::isinf(x)) return x > 0 ? FLT_MAX : -INFINITY;
  if ((double)f > x) f = std::nextafter(f, -INFINITY);
  return f;
}

float d2f_ru(double x)
{
  if (std::isnan(x)) return (float)x;
  float f = (float)x;
  if (std::isinf(f) && !std::isinf(x)) return x < 0 ? -FLT_MAX : INFINITY;
  if ((double)f < x) f = std::nextafter(f, INFINITY);
  return f;
}

// FP64 -> FP32 rounded to nearest, ties to even, whatever the host's
// current rounding mode
float d2f_rn(double x)
{
  const float lo = d2f_rd(x), hi = d2f_ru(x);
  if (lo == hi || std::isnan(x)) return lo;
  const double dl = x - (double)lo, dh = (double)hi - x;
  if (dl != dh) return dl < dh ? lo : hi;
  uint32_t bits;
  std::memcpy(&bits, &lo, 4);
  return (bits & 1u) ? hi : lo;
}

static bool is_unary(int op)
{
  return op == CMN_OP_SQR || op == CMN_OP_NEG || op == CMN_OP_EXP || op == CMN_OP_LOG || op == CMN_OP_SQRT ||
         op == CMN_OP_SIN || op == CMN_OP_COS || op == CMN_OP_TANH || op == CMN_OP_POWN || op == CMN_OP_ABS;
}

static bool interval_op(int op)
{
  switch (op) {
    case CMN_OP_ADD: case CMN_OP_SUB: case CMN_OP_MUL: case CMN_OP_DIV: case CMN_OP_SQR:
    case CMN_OP_NEG: case CMN_OP_SQRT: case CMN_OP_POWN: case CMN_OP_ABS: case CMN_OP_MIN:
    case CMN_OP_MAX: case CMN_OP_EXP: case CMN_OP_LOG: case CMN_OP_SIN: case CMN_OP_COS:
    case CMN_OP_TANH: case CMN_OP_POW:
      return true;
    default:
      return false;
  }
}

static const char* op_name(int op)
{
  static const char* names[] = {"Var", "Const", "Add", "Sub", "Mul", "Div", "Sqr", "Neg", "Exp", "Log",
                                "Sqrt", "Sin", "Cos", "Tanh", "PowN", "Pow", "Abs", "Min", "Max"};
  return (op >= 0 && op <= 18) ? names[op] : "?";
}

cmn_status build_host_problem(const cmn_problem_desc* d, HostProblem& p, std::string& err)
{
  if (d == nullptr || d->nodes == nullptr || d->n_nodes <= 0) {
    err = "empty DAG";
    return CMN_INVALID_DAG;
  }
  p.nodes.assign(d->nodes, d->nodes + d->n_nodes);
  if (d->n_vars > 0) {
    if (!d->var_lb || !d->var_ub || !d->var_kinds) {
      err = "missing variable bounds or kinds";
      return CMN_INVALID_PROBLEM;
    }
    p.var_lb.assign(d->var_lb, d->var_lb + d->n_vars);
    p.var_ub.assign(d->var_ub, d->var_ub + d->n_vars);
    p.var_kinds.assign(d->var_kinds, d->var_kinds + d->n_vars);
  }
  if (d->n_constraints > 0) {
    if (!d->constraints) {
      err = "missing constraints";
      return CMN_INVALID_PROBLEM;
    }
    p.constraints.assign(d->constraints, d->constraints + d->n_constraints);
  }
  p.objective_root = d->objective_root;
  const int64_t n = (int64_t)p.nodes.size();

  // graph bookkeeping (model/problem.hpp:286-307)
  int64_t var_nodes = 0;
  for (int64_t i = 0; i < n; ++i) {
    const cmn_node& nd = p.nodes[i];
    if (nd.op < 0 || nd.op > CMN_OP_MAX) {
      err = "node " + std::to_string(i) + " has an unknown op";
      return CMN_INVALID_DAG;
    }
    const int need = (nd.op == CMN_OP_VAR || nd.op == CMN_OP_CONST) ? 0 : (is_unary(nd.op) ? 1 : 2);
    if (nd.n_in != need) {
      err = "node " + std::to_string(i) + " (" + op_name(nd.op) + ") has " + std::to_string(nd.n_in) +
            " operands, expected " + std::to_string(need);
      return CMN_INVALID_DAG;
    }
    if ((need >= 1 && (nd.in0 < 0 || nd.in0 >= i)) || (need >= 2 && (nd.in1 < 0 || nd.in1 >= i))) {
      err = "DAG node operand id is not strictly less than the node's own id; topological-order invariant "
            "violated";
      return CMN_INVALID_DAG;
    }
    if (nd.op == CMN_OP_VAR) {
      if (nd.var_index != var_nodes) {
        err = "Var nodes must carry var_index 0, 1, ... in node order";
        return CMN_INVALID_DAG;
      }
      ++var_nodes;
    }
    if (nd.op == CMN_OP_POWN && (nd.int_exp < -32768 || nd.int_exp > 32767)) {
      err = "PowN exponent out of range";
      return CMN_INVALID_DAG;
    }
  }
  if (var_nodes != (int64_t)p.var_lb.size()) {
    err = "box_bounds/var_kinds are out of sync with the number of Op::Var nodes";
    return CMN_INVALID_DAG;
  }
  if (p.objective_root >= 0 && p.objective_root < n && p.nodes[p.objective_root].op == CMN_OP_CONST) {
    err = "objective root is a bare Const; set_objective was given a fixed() value rather than an expression to "
          "optimise";
    return CMN_INVALID_DAG;
  }
  for (const auto& c : p.constraints) {
    if (c.root < 0 || c.root >= n) {
      err = "constraint root out of range";
      return CMN_INVALID_DAG;
    }
    if (p.nodes[c.root].op == CMN_OP_CONST) {
      err = "constraint root is a bare Const; add_constraint was given a fixed() value rather than an expression";
      return CMN_INVALID_DAG;
    }
    if (c.cmp != CMN_CMP_LE && c.cmp != CMN_CMP_EQ) {
      err = "constraint comparison must be LE or EQ";
      return CMN_INVALID_PROBLEM;
    }
  }
  // problem-level checks (model/problem.hpp:324-354)
  if (p.var_lb.empty()) {
    err = "Problem has zero variables";
    return CMN_INVALID_PROBLEM;
  }
  if (p.objective_root < 0 || p.objective_root >= n) {
    err = "Problem's objective was never set (set_objective was never called)";
    return CMN_INVALID_PROBLEM;
  }
  for (size_t i = 0; i < p.var_lb.size(); ++i) {
    const double lb = p.var_lb[i], ub = p.var_ub[i];
    if (!(lb <= ub)) {
      err = "variable's lower bound exceeds its upper bound";
      return CMN_INVALID_PROBLEM;
    }
    const int k = p.var_kinds[i];
    if (k != CMN_VAR_CONTINUOUS && k != CMN_VAR_INTEGER && k != CMN_VAR_BINARY) {
      err = "unknown variable kind";
      return CMN_INVALID_PROBLEM;
    }
    if (k == CMN_VAR_INTEGER || k == CMN_VAR_BINARY) {
      if (std::floor(lb) < lb || std::floor(ub) < ub) {
        err = "Integer/Binary variable has non-integer-valued bounds";
        return CMN_INVALID_PROBLEM;
      }
    }
    if (k == CMN_VAR_BINARY && (lb < 0 || lb > 0 || ub < 1 || ub > 1)) {
      err = "Binary variable's bounds are not exactly [0,1]";
      return CMN_INVALID_PROBLEM;
    }
  }
  for (const auto& c : p.constraints) {
    if (!std::isfinite(c.rhs)) {
      err = "constraint rhs must be finite";
      return CMN_INVALID_PROBLEM;
    }
  }
  if (p.var_lb.size() > 60000) {
    err = "more than 60000 variables";
    return CMN_INVALID_PROBLEM;
  }

  // reachability (backend/graph/cost.hpp:38-68)
  p.reach.assign(n, 0);
  p.reach[p.objective_root] = 1;
  for (const auto& c : p.constraints) p.reach[c.root] = 1;
  p.buffer_node_count = 0;
  for (int64_t i = n - 1; i >= 0; --i) {
    if (!p.reach[i]) continue;
    const cmn_node& nd = p.nodes[i];
    if (nd.n_in >= 1) p.reach[nd.in0] = 1;
    if (nd.n_in >= 2) p.reach[nd.in1] = 1;
    if (nd.op != CMN_OP_CONST) ++p.buffer_node_count;
  }
  for (int64_t i = 0; i < n; ++i) {
    if (!p.reach[i]) continue;
    const cmn_node& nd = p.nodes[i];
    if ((is_unary(nd.op)) && p.nodes[nd.in0].op == CMN_OP_CONST) {
      err = std::string(op_name(nd.op)) + " applied directly to an Op::Const";
      return CMN_INVALID_DAG;
    }
  }
  return CMN_OK;
}

namespace {

enum State : uint8_t { kNone, kVarS, kConstS, kSlotS, kAccS, kDeferred, kAbsorbed };

struct TermForm {
  bool ok = false;
  uint8_t pkind = 0;  // kTermProd / kTermSqr / kTermVar
  bool has_c = false;
  double c = 0;
  uint16_t a = 0, b = 0;
  int64_t inner = -1;  // absorbed product node, if any
};

class Compiler {
 public:
  Compiler(const HostProblem& p, Program& out) : p_(p), out_(out) {}

  void run()
  {
    const int64_t n = (int64_t)p_.nodes.size();
    uses_.assign(n, 0);
    state_.assign(n, kNone);
    slot_of_.assign(n, -1);
    form_.assign(n, TermForm{});
    consumer_.assign(n, -1);
    for (int64_t i = 0; i < n; ++i) {
      if (!p_.reach[i]) continue;
      const cmn_node& nd = p_.nodes[i];
      if (nd.n_in >= 1) {
        ++uses_[nd.in0];
        consumer_[nd.in0] = i;
      }
      if (nd.n_in >= 2) {
        ++uses_[nd.in1];
        consumer_[nd.in1] = i;
      }
    }
    ++uses_[p_.objective_root];
    for (const auto& c : p_.constraints) ++uses_[c.root];
    // roots are consumed by their checks, never by a chain
    is_root_.assign(n, 0);
    is_root_[p_.objective_root] = 1;
    for (const auto& c : p_.constraints) is_root_[c.root] = 1;

    // algorithmic op counts (weights: add/sub 2, scalar*interval 2,
    // interval*interval 8, sqr 2, neg 0, feasibility 1 compare)
    for (int64_t i = 0; i < n; ++i) {
      if (!p_.reach[i]) continue;
      const cmn_node& nd = p_.nodes[i];
      switch (nd.op) {
        case CMN_OP_VAR: case CMN_OP_CONST: break;
        case CMN_OP_ADD: case CMN_OP_SUB: out_.flops_per_box += 2; out_.point_flops_per_box += 1; break;
        case CMN_OP_MUL: {
          const bool sc = p_.nodes[nd.in0].op == CMN_OP_CONST || p_.nodes[nd.in1].op == CMN_OP_CONST;
          out_.flops_per_box += sc ? 2 : 8;
          out_.point_flops_per_box += 1;
          break;
        }
        case CMN_OP_SQR: out_.flops_per_box += 2; out_.point_flops_per_box += 1; break;
        case CMN_OP_NEG: break;
        case CMN_OP_DIV: out_.flops_per_box += 8; out_.point_flops_per_box += 1; break;
        default: out_.flops_per_box += 2; out_.point_flops_per_box += 1; break;
      }
      if (!(nd.op == CMN_OP_VAR || nd.op == CMN_OP_CONST) && !interval_op(nd.op) && out_.interval_supported) {
        out_.interval_supported = false;
        out_.unsupported_op = op_name(nd.op);
      }
    }
    out_.flops_per_box += (double)p_.constraints.size();
    out_.point_flops_per_box += (double)p_.constraints.size();

    classify_terms();
    emit_all();
    out_.n_slots = max_slots_;
    build_schedule();
    build_incremental();
    build_chains();
    build_levels();
    out_.code32 = out_.code64;
    out_.code32p = out_.code64;
    for (size_t k = 0; k < out_.code64.size(); ++k) {
      Instr& s = out_.code32[k];
      Instr& q = out_.code32p[k];
      const Instr& d = out_.code64[k];
      const int code = d.head & 7;
      if (code == kOpCheck) continue;  // rhs stays FP64
      const bool has_const = code == kOpTerm || code == kOpConstToSlot ||
                             (code == kOpGeneric && ((d.modes & 3) == kModeConst || ((d.modes >> 2) & 3) == kModeConst)) ||
                             (code == kOpLoadAcc && (d.modes & 3) == kModeConst) ||
                             (code == kOpObjective && (d.modes & 3) == kModeConst);
      if (has_const) {
        const double c = d.c;
        s.c32.clo = d2f_rd(c);
        s.c32.chi = d2f_ru(c);
        q.c32.clo = d2f_rn(c);
        q.c32.chi = q.c32.clo;
      }
    }
    out_.code32l = out_.code64l;
    for (size_t k = 0; k < out_.code64l.size(); ++k) {  // the same constants, the levels' slots
      const Instr l = out_.code64l[k];
      Instr& s = out_.code32l[k];
      s = out_.code32[k];
      s.dst = l.dst;
      s.a = l.a;
      s.b = l.b;
    }
  }

 private:
  // Splits a slot-free program at every accumulator reset (a chain's first
  // TERM, or LoadAcc) into independent segments, then assigns them to the
  // lanes of groups of 2..32 lanes, longest first, each to the lane with
  // the least work so far.
  void build_schedule()
  {
    const int len = (int)out_.code64.size();
    if (out_.n_slots != 0 || len == 0) return;
    std::vector<std::pair<int, int>> segs;
    int start = 0;
    for (int pc = 1; pc < len; ++pc) {
      const Instr& in = out_.code64[pc];
      const int code = in.head & 7, sub = in.head >> 3;
      if ((code == kOpTerm && (sub & kTermInit)) || code == kOpLoadAcc) {
        segs.push_back({start, pc});
        start = pc;
      }
    }
    segs.push_back({start, len});
    // a point stops at its first violated constraint: the segments that
    // hold the objective come last in every lane's list (level 0: one lane,
    // program order otherwise)
    auto holds_objective = [&](const std::pair<int, int>& sg) {
      for (int pc = sg.first; pc < sg.second; ++pc)
        if ((out_.code64[pc].head & 7) == kOpObjective) return true;
      return false;
    };
    const std::vector<std::pair<int, int>> in_order = segs;
    std::stable_sort(segs.begin(), segs.end(), [](const std::pair<int, int>& a, const std::pair<int, int>& b) {
      return (a.second - a.first) > (b.second - b.first);
    });
    const int ns = (int)segs.size();
    out_.n_segments = ns;
    out_.sched.assign(6, 0);
    out_.makespan.assign(6, 0);
    out_.makespan[0] = len;
    out_.sched[0] = (int32_t)out_.sched.size();
    out_.sched.push_back(0);
    out_.sched.push_back(ns);
    for (int pass = 0; pass < 2; ++pass)
      for (const auto& sg : in_order)
        if (holds_objective(sg) == (pass == 1)) {
          out_.sched.push_back(sg.first);
          out_.sched.push_back(sg.second);
        }
    for (int l = 1; l <= 5; ++l) {
      const int G = 1 << l;
      std::vector<std::vector<int>> lanes(G);
      std::vector<int64_t> load(G, 0);
      for (int j = 0; j < ns; ++j) {
        int best = 0;
        for (int q = 1; q < G; ++q)
          if (load[q] < load[best]) best = q;
        lanes[best].push_back(j);
        load[best] += segs[j].second - segs[j].first;
      }
      out_.makespan[l] = *std::max_element(load.begin(), load.end());
      out_.sched[l] = (int32_t)out_.sched.size();
      int32_t acc = 0;
      out_.sched.push_back(0);
      for (int q = 0; q < G; ++q) {
        acc += (int32_t)lanes[q].size();
        out_.sched.push_back(acc);
      }
      for (int q = 0; q < G; ++q)
        for (int pass = 0; pass < 2; ++pass)
          for (int j : lanes[q])
            if (holds_objective(segs[j]) == (pass == 1)) {
              out_.sched.push_back(segs[j].first);
              out_.sched.push_back(segs[j].second);
            }
    }
    // more lanes per box only while they cut the busiest lane's work by a
    // fifth or more
    out_.group_max = 1;
    for (int l = 1; l <= 5; ++l) {
      if (out_.makespan[l] * 5 > out_.makespan[l - 1] * 4) break;
      out_.group_max = 1 << l;
    }
  }

  // Segments of a slot-free program as sum chains plus their readers, and
  // per (variable, segment) the chain instructions that read the variable
  // (Program::inc_*).  Leaves inc_ok false for any other shape.
  void build_incremental()
  {
    const std::vector<Instr>& code = out_.code64;
    const int len = (int)code.size();
    const int n = (int)p_.n_vars();
    if (out_.n_slots != 0 || len == 0) return;
    auto accumulates = [](const Instr& in) {
      const int code = in.head & 7;
      return code == kOpTerm || code == kOpLoadAcc;
    };
    auto starts = [](const Instr& in) {
      const int code = in.head & 7, sub = in.head >> 3;
      return (code == kOpTerm && (sub & kTermInit)) || code == kOpLoadAcc;
    };
    std::vector<int32_t> seg;
    int pc = 0;
    while (pc < len) {
      const int b = pc;
      int t = pc;
      if (starts(code[pc])) {
        t = pc + 1;
        while (t < len && accumulates(code[t]) && !starts(code[t])) ++t;
      }
      int e = t;
      while (e < len && !accumulates(code[e])) {
        const int c = code[e].head & 7;
        if (c != kOpCheck && c != kOpObjective) return;  // slots or other forms
        ++e;
      }
      if (e == b) return;  // an accumulating instruction that does not start a chain
      seg.push_back(b);
      seg.push_back(t);
      seg.push_back(e);
      pc = e;
    }
    const int S = (int)seg.size() / 3;
    std::vector<std::vector<int32_t>> lists((size_t)n * S);
    for (int s = 0; s < S; ++s) {
      for (int q = seg[3 * s]; q < seg[3 * s + 1]; ++q) {
        const Instr& in = code[q];
        const int c = in.head & 7;
        int va = -1, vb = -1;
        if (c == kOpTerm) {
          va = in.a;
          vb = in.b;
        } else if ((in.modes & 3) == kModeVar) {  // LoadAcc of a variable
          va = vb = in.a;
        }
        if (va >= n || vb >= n) return;
        if (va >= 0) lists[(size_t)va * S + s].push_back(q);
        if (vb >= 0 && vb != va) lists[(size_t)vb * S + s].push_back(q);
      }
    }
    out_.inc_seg = seg;
    out_.inc_segments = S;
    out_.inc_off.assign((size_t)n * S + 1, 0);
    out_.inc_pcs.clear();
    for (size_t i = 0; i < lists.size(); ++i) {
      out_.inc_off[i] = (int32_t)out_.inc_pcs.size();
      out_.inc_pcs.insert(out_.inc_pcs.end(), lists[i].begin(), lists[i].end());
    }
    out_.inc_off[lists.size()] = (int32_t)out_.inc_pcs.size();
    out_.inc_ok = true;
  }

  // Program::level_*.
  void build_levels()
  {
    const std::vector<Instr>& code = out_.code64;
    const int len = (int)code.size();
    if (out_.n_slots == 0 || len < 4 * kLevelWarps) return;
    auto is = [&](int pc, int op) { return (code[pc].head & 7) == op; };
    auto resets = [&](int pc) { return is(pc, kOpLoadAcc) || (is(pc, kOpTerm) && ((code[pc].head >> 3) & kTermInit)); };
    // which operand fields an instruction reads, and whether it reads the accumulator
    auto slots_of = [&](int pc, int (&s)[2]) {
      const Instr& in = code[pc];
      const int ma = in.modes & 3, mb = (in.modes >> 2) & 3;
      s[0] = s[1] = -1;
      if (is(pc, kOpTerm) || is(pc, kOpStoreAcc) || is(pc, kOpConstToSlot)) return;
      if (ma == kModeSlot) s[0] = in.a;
      if (is(pc, kOpGeneric) && mb == kModeSlot) s[1] = in.b;
    };
    auto reads_acc = [&](int pc) {
      const Instr& in = code[pc];
      const int sub = in.head >> 3;
      if (is(pc, kOpStoreAcc)) return true;
      if (is(pc, kOpTerm)) return !(sub & kTermInit);
      if (is(pc, kOpConstToSlot)) return false;
      if ((in.modes & 3) == kModeAcc) return true;
      // a unary node's second operand points at the accumulator unread
      const bool binary = is(pc, kOpGeneric) && (sub == kGAdd || sub == kGSub || sub == kGMul || sub == kGDiv ||
                                                 sub == kGPow || sub == kGMin || sub == kGMax);
      return binary && ((in.modes >> 2) & 3) == kModeAcc;
    };
    auto writes = [&](int pc) { return is(pc, kOpGeneric) || is(pc, kOpStoreAcc) || is(pc, kOpConstToSlot); };
    // runs: from an accumulator reset to its last reader, else one instruction
    std::vector<std::pair<int, int>> runs;
    for (int pc = 0; pc < len;) {
      int end = pc + 1;
      if (resets(pc)) {
        for (int q = pc + 1; q < len && !resets(q); ++q)
          if (reads_acc(q)) end = q + 1;
      } else if (reads_acc(pc)) {
        return;  // an accumulator read outside its chain's run: never emitted
      }
      runs.push_back({pc, end});
      pc = end;
    }
    // levels: one past the runs that wrote the slots a run reads
    const int R = (int)runs.size();
    std::vector<int> writer(out_.n_slots, -1), level(R, 0);
    std::vector<std::vector<int>> values(R);           // instructions of a run that write slots
    std::vector<std::array<int, 2>> from(len, {-1, -1});  // instruction that wrote each operand
    std::vector<int> run_of(len, 0), def(out_.n_slots, -1);
    int levels = 0;
    for (int r = 0; r < R; ++r) {
      for (int pc = runs[r].first; pc < runs[r].second; ++pc) {
        run_of[pc] = r;
        int s[2];
        slots_of(pc, s);
        for (int e = 0; e < 2; ++e) {
          if (s[e] < 0) continue;
          const int d = def[s[e]];
          if (d < 0) return;  // a slot read before it is written: never emitted
          from[pc][e] = d;
          if (run_of[d] != r) level[r] = std::max(level[r], level[run_of[d]] + 1);
        }
        if (writes(pc)) def[code[pc].dst] = pc;
      }
      levels = std::max(levels, level[r] + 1);
    }
    // warps: longest run first, to the warp with the least of the level
    std::vector<std::vector<std::vector<int>>> lists(levels, std::vector<std::vector<int>>(kLevelWarps));
    std::vector<int> order(R);
    for (int r = 0; r < R; ++r) order[r] = r;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
      return runs[a].second - runs[a].first > runs[b].second - runs[b].first;
    });
    std::vector<std::array<int, kLevelWarps>> load(levels);
    for (auto& l : load) l.fill(0);
    for (int r : order) {
      int w = 0;
      for (int q = 1; q < kLevelWarps; ++q)
        if (load[level[r]][q] < load[level[r]][w]) w = q;
      lists[level[r]][w].push_back(r);
      load[level[r]][w] += runs[r].second - runs[r].first;
    }
    int64_t span = 0;
    for (const auto& l : load) span += *std::max_element(l.begin(), l.end());
    if (span * 2 > len) return;  // too sequential for the barriers to pay
    // slots: a value keeps its own from its level to the last one that reads it
    std::vector<int> last(len, -1), slot(len, -1), free_list;
    for (int pc = 0; pc < len; ++pc)
      for (int e = 0; e < 2; ++e)
        if (from[pc][e] >= 0) last[from[pc][e]] = std::max(last[from[pc][e]], level[run_of[pc]]);
    std::vector<std::vector<int>> dies(levels);
    int next = 0;
    for (int l = 0; l < levels; ++l) {
      for (int w = 0; w < kLevelWarps; ++w)
        for (int r : lists[l][w])
          for (int pc = runs[r].first; pc < runs[r].second; ++pc)
            if (writes(pc)) {
              if (free_list.empty()) free_list.push_back(next++);
              slot[pc] = free_list.back();
              free_list.pop_back();
              dies[std::max(last[pc], l)].push_back(slot[pc]);
            }
      free_list.insert(free_list.end(), dies[l].begin(), dies[l].end());
    }
    out_.level_slots = next;
    out_.code64l = code;
    for (int pc = 0; pc < len; ++pc) {
      Instr& in = out_.code64l[pc];
      if (writes(pc)) in.dst = (uint16_t)slot[pc];
      if (from[pc][0] >= 0) in.a = (uint16_t)slot[from[pc][0]];
      if (from[pc][1] >= 0) in.b = (uint16_t)slot[from[pc][1]];
    }
    for (int l = 0; l < levels; ++l)
      for (int w = 0; w < kLevelWarps; ++w) {
        out_.level_off.push_back((int32_t)out_.level_run.size() / 2);
        for (int r : lists[l][w]) {
          out_.level_run.push_back(runs[r].first);
          out_.level_run.push_back(runs[r].second);
        }
      }
    out_.level_off.push_back((int32_t)out_.level_run.size() / 2);
  }

  // Most that the FP32 filter of a chain of k terms can be off its FP64
  // lower bound, per unit of summed term magnitude.  Per term: the two
  // bounds cut to FP32 (2 u each, u = 2^-24), the product, the coefficient
  // and its product (u each), 7 u.  The sum: two interleaved accumulators of
  // k / 2 adds, joined, plus the constant: (k / 2 + 2) u.  The FP64 chain's
  // own roundings (2^-52 each) and the comparison take the rest of the 13.
  // The factor covers the products of these and the error of the summed
  // magnitude itself (k / 2 u, k <= 8192).
  static float chain_eps(int64_t k) { return (float)((double)(k / 2 + 13) * std::ldexp(1.0, -24) * 1.02); }

  // Program::chain_*: the incremental segments as chains by reader.
  void build_chains()
  {
    if (!out_.inc_ok) return;
    const std::vector<Instr>& code = out_.code64;
    std::vector<ChainSeg> segs;
    for (int s = 0; s < out_.inc_segments; ++s) {
      ChainSeg cs;
      std::memset(&cs, 0, sizeof cs);
      cs.kind = kChainGeneral;
      cs.pc0 = out_.inc_seg[3 * s];
      cs.pc1 = out_.inc_seg[3 * s + 1];
      cs.pc2 = out_.inc_seg[3 * s + 2];
      if (cs.pc1 > cs.pc0 && cs.pc2 == cs.pc1 + 1) {
        const Instr& rd = code[cs.pc1];
        const int op = rd.head & 7;
        if ((rd.modes & 3) == kModeAcc && op == kOpObjective) cs.kind = kChainObjective;
        if ((rd.modes & 3) == kModeAcc && op == kOpCheck) {
          if ((rd.head >> 3) == CMN_CMP_LE) cs.kind = kChainLe;
          else cs.eq = 1;
          cs.rhs = rd.c;
          cs.rhs_dn = d2f_rd(rd.c);
          cs.rhs_up = d2f_ru(rd.c);
        }
      }
      if (cs.kind != kChainGeneral || cs.eq) add_filter(cs);
      segs.push_back(cs);
    }
    auto rank = [&](const ChainSeg& s) {  // the objective's chain, general ones, <= chains
      for (int pc = s.pc1; pc < s.pc2; ++pc)
        if ((code[pc].head & 7) == kOpObjective) return -1;
      return (int)s.kind;
    };
    std::stable_sort(segs.begin(), segs.end(), [&](const ChainSeg& a, const ChainSeg& b) {
      const int ra = rank(a), rb = rank(b);
      return ra != rb ? ra < rb : a.pc1 - a.pc0 > b.pc1 - b.pc0;
    });
    out_.chain_seg = segs;
    for (const Instr& in : code)
      if ((in.head & 7) == kOpTerm && ((in.head >> 3) & kTermPMask) != kTermVar) ++out_.chain_products;
    build_chains32();
    build_point_chains();
    out_.chain_points = !segs.empty() && segs[0].kind == kChainObjective;
    for (const ChainSeg& s : segs) out_.chain_points = out_.chain_points && s.eps > 0.0f;
    for (size_t v = 0; v < p_.var_lb.size(); ++v)
      out_.chain_points =
          out_.chain_points && std::fabs(p_.var_lb[v]) <= kFilterMax && std::fabs(p_.var_ub[v]) <= kFilterMax;
  }

  // Program::chain_term_pt: the chains' terms for FP32 points, for programs
  // of one objective chain and single <= or == checks.
  void build_point_chains()
  {
    const uint32_t one = (uint32_t)p_.var_lb.size();
    if (one > 0xffffu || out_.chain_seg.empty() || out_.chain_seg[0].kind != kChainObjective) return;
    for (const ChainSeg& s : out_.chain_seg)
      if (s.kind == kChainGeneral && !s.eq) return;
    for (ChainSeg& cs : out_.chain_seg) {
      cs.pt = (int32_t)out_.chain_term_pt.size();
      for (int pc = cs.pc0; pc < cs.pc1; ++pc) {
        const Instr& in = out_.code64[pc];
        const int sub = in.head >> 3, pk = sub & kTermPMask;
        ChainTerm t = {one | (one << 16), 1.0f};
        if ((in.head & 7) == kOpLoadAcc) {
          if ((in.modes & 3) == kModeVar) t.ab = in.a | (one << 16);
          else t.c = d2f_rn(in.c);
        } else {
          t.ab = in.a | ((pk == kTermProd ? (uint32_t)in.b : pk == kTermSqr ? (uint32_t)in.a : one) << 16);
          if (sub & kTermHasC) t.c = d2f_rn(in.c);
          if ((sub & kTermSub) && !(sub & kTermInit)) t.c = -t.c;
        }
        out_.chain_term_pt.push_back(t);
      }
      cs.pt_end = (int32_t)out_.chain_term_pt.size();
    }
  }

  // Program::chain_term32 and chain_var32: the chains' terms with outward FP32
  // coefficients, whole and by variable.
  void build_chains32()
  {
    const size_t n = p_.var_lb.size(), S = out_.chain_seg.size();
    if (n + 1 > 0xffff) return;
    std::vector<std::pair<size_t, ChainTerm32>> by_var;  // (variable, chain) of each term read, in program order
    std::vector<ChainTerm32> all;
    for (size_t q = 0; q < S; ++q) {
      ChainSeg& cs = out_.chain_seg[q];
      if (cs.kind == kChainGeneral) return;
      cs.t32 = (int32_t)all.size();
      for (int pc = cs.pc0; pc < cs.pc1; ++pc) {
        const Instr& in = out_.code64[pc];
        const int sub = in.head >> 3, pk = sub & kTermPMask;
        ChainTerm32 t;
        std::memset(&t, 0, sizeof t);
        if ((in.head & 7) == kOpLoadAcc && (in.modes & 3) != kModeVar) {
          t.flags = kT32Const;
          t.cl = d2f_rd(in.c);
          t.ch = d2f_ru(in.c);
          if (!std::isfinite(t.cl) || !std::isfinite(t.ch)) return;
          all.push_back(t);
          continue;
        }
        const bool term = (in.head & 7) == kOpTerm, has_c = term && (sub & kTermHasC);
        const bool subtracts = term && (sub & kTermSub) && !(sub & kTermInit);
        const double c = has_c ? in.c : 1.0;
        if (!(std::fabs(c) >= std::ldexp(1.0, -40) && std::fabs(c) <= std::ldexp(1.0, 40))) return;
        t.cl = d2f_rd(std::fabs(c));
        t.ch = d2f_ru(std::fabs(c));
        if ((c < 0.0) != subtracts) t.flags |= kT32Neg;
        if (subtracts) t.flags |= kT32Sub;
        uint32_t a = in.a, b = (uint32_t)n;
        if (term && pk == kTermProd) b = in.b;
        else if (term && pk == kTermSqr) t.flags |= kT32Sqr, b = in.a;
        else if (!has_c) t.flags |= kT32Raw;
        t.ab = a | (b << 16);
        all.push_back(t);
        by_var.push_back({a * S + q, t});
        if (b != a && b < n) {
          t.ab = b | (a << 16);
          by_var.push_back({b * S + q, t});
        }
      }
      cs.t32_end = (int32_t)all.size();
    }
    out_.chain_term32 = all;
    std::vector<int32_t>& off = out_.chain_var_off;  // by counting: a list per pair took 13 % of 1,500 x 1,500
    off.assign(n * S + 1, 0);
    for (const auto& e : by_var) ++off[e.first + 1];
    for (size_t i = 0; i < n * S; ++i) off[i + 1] += off[i];
    std::vector<int32_t> at(off.begin(), off.end() - 1);
    out_.chain_var32.resize(by_var.size());
    for (const auto& e : by_var) out_.chain_var32[at[e.first]++] = e.second;
  }

  // The FP32 filter's terms of a chain; leaves eps 0 (no filter) when a
  // coefficient is outside the range its error bound covers.
  void add_filter(ChainSeg& cs)
  {
    auto in_range = [](double c) { return std::fabs(c) >= std::ldexp(1.0, -40) && std::fabs(c) <= std::ldexp(1.0, 40); };
    std::vector<ChainTerm> groups[6];
    bool ok = cs.pc1 - cs.pc0 <= 8192;
    auto put = [&](int g, double c, uint32_t a, uint32_t b) {
      if (c == 0.0) return;
      ok = ok && in_range(c);
      groups[g + (c < 0.0 ? 1 : 0)].push_back(ChainTerm{a | (b << 16), d2f_rn(c)});
    };
    for (int pc = cs.pc0; pc < cs.pc1; ++pc) {
      const Instr& in = out_.code64[pc];
      const int sub = in.head >> 3;
      if ((in.head & 7) == kOpLoadAcc) {
        if ((in.modes & 3) == kModeVar) put(4, 1.0, in.a, in.a);
        else if (in.c == 0.0 || in_range(in.c)) cs.c0 = d2f_rn(in.c);
        else ok = false;
        continue;
      }
      const double c = (sub & kTermHasC) ? in.c : 1.0;
      const double sc = ((sub & kTermSub) && !(sub & kTermInit)) ? -c : c;
      const int pk = sub & kTermPMask;
      put(pk == kTermProd ? 0 : pk == kTermSqr ? 2 : 4, sc, in.a, pk == kTermProd ? in.b : in.a);
    }
    int64_t k = 0;
    for (int g = 0; g < 6; ++g) {
      cs.group[g] = (int32_t)out_.chain_term.size();
      out_.chain_term.insert(out_.chain_term.end(), groups[g].begin(), groups[g].end());
      if (out_.chain_term.size() & 1) out_.chain_term.push_back(ChainTerm{0, 0.0f});
      k += (int64_t)groups[g].size() + 1;
    }
    cs.group[6] = (int32_t)out_.chain_term.size();
    cs.eps = ok ? chain_eps(k) : 0.0f;
  }

  bool is_var(int64_t id) const { return p_.nodes[id].op == CMN_OP_VAR; }
  bool is_const(int64_t id) const { return p_.nodes[id].op == CMN_OP_CONST; }

  // P-form of a node built only from variables: x*y, sqr(x), x.
  bool pform(int64_t id, uint8_t& pk, uint16_t& a, uint16_t& b) const
  {
    const cmn_node& nd = p_.nodes[id];
    if (nd.op == CMN_OP_VAR) {
      pk = kTermVar;
      a = b = (uint16_t)nd.var_index;
      return true;
    }
    if (nd.op == CMN_OP_MUL && is_var(nd.in0) && is_var(nd.in1)) {
      pk = kTermProd;
      a = (uint16_t)p_.nodes[nd.in0].var_index;
      b = (uint16_t)p_.nodes[nd.in1].var_index;
      return true;
    }
    if (nd.op == CMN_OP_SQR && is_var(nd.in0)) {
      pk = kTermSqr;
      a = b = (uint16_t)p_.nodes[nd.in0].var_index;
      return true;
    }
    return false;
  }

  // A node whose single consumer is an Add/Sub and whose value is c*P or P
  // is evaluated inside that consumer's term instruction (deferred); the
  // inner P of a c*P term is absorbed into it.
  void classify_terms()
  {
    const int64_t n = (int64_t)p_.nodes.size();
    for (int64_t i = 0; i < n; ++i) {
      if (!p_.reach[i] || is_var(i) || is_const(i)) continue;
      if (uses_[i] != 1 || is_root_[i]) continue;
      const int64_t cons = consumer_[i];
      if (cons < 0) continue;
      const int cop = p_.nodes[cons].op;
      if (cop != CMN_OP_ADD && cop != CMN_OP_SUB) continue;
      const cmn_node& nd = p_.nodes[i];
      TermForm f;
      uint8_t pk;
      uint16_t a, b;
      if (nd.op == CMN_OP_MUL && (is_const(nd.in0) != is_const(nd.in1))) {
        const int64_t c_id = is_const(nd.in0) ? nd.in0 : nd.in1;
        const int64_t x_id = is_const(nd.in0) ? nd.in1 : nd.in0;
        if (pform(x_id, pk, a, b) && (is_var(x_id) || (uses_[x_id] == 1 && !is_root_[x_id]))) {
          f.ok = true;
          f.pkind = pk;
          f.has_c = true;
          f.c = p_.nodes[c_id].constant;
          f.a = a;
          f.b = b;
          f.inner = is_var(x_id) ? -1 : x_id;
        }
      } else if (pform(i, pk, a, b)) {
        f.ok = true;
        f.pkind = pk;
        f.a = a;
        f.b = b;
      }
      if (f.ok) {
        form_[i] = f;
        state_[i] = kDeferred;
        if (f.inner >= 0) state_[f.inner] = kAbsorbed;
      }
    }
  }

  int alloc_slot()
  {
    int s;
    if (!free_slots_.empty()) {
      // lowest free slot keeps the working set compact
      auto it = std::min_element(free_slots_.begin(), free_slots_.end());
      s = *it;
      free_slots_.erase(it);
    } else {
      s = next_slot_++;
    }
    max_slots_ = std::max(max_slots_, s + 1);
    return s;
  }

  void consume(int64_t id)
  {
    if (--uses_[id] == 0) {
      if (state_[id] == kSlotS && slot_of_[id] >= 0) {
        free_slots_.push_back(slot_of_[id]);
        slot_of_[id] = -1;
      }
      if (state_[id] == kAccS && acc_holder_ == id) acc_holder_ = -1;
    }
  }

  void emit(const Instr& ins) { out_.code64.push_back(ins); }

  static Instr blank()
  {
    Instr ins;
    std::memset(&ins, 0, sizeof ins);
    return ins;
  }

  // Frees the accumulator: a live value held there moves to a slot.
  void spill_acc()
  {
    if (acc_holder_ < 0) return;
    const int64_t h = acc_holder_;
    acc_holder_ = -1;
    if (uses_[h] <= 0) return;
    const int s = alloc_slot();
    Instr ins = blank();
    ins.head = make_head(kOpStoreAcc, 0);
    ins.dst = (uint16_t)s;
    emit(ins);
    state_[h] = kSlotS;
    slot_of_[h] = s;
  }

  // Ensures `id` is readable as an operand (slot, var, const or acc).
  void materialise(int64_t id)
  {
    if (state_[id] == kDeferred || state_[id] == kAbsorbed) {
      const TermForm f = form_[id];
      if (state_[id] == kDeferred && f.ok) {
        // evaluate the term generically: P into a slot, then c*P
        if (f.inner >= 0) materialise(f.inner);
        const cmn_node& nd = p_.nodes[id];
        emit_generic(id, nd);
        return;
      }
      emit_generic(id, p_.nodes[id]);
    }
  }

  void operand(int64_t id, uint8_t& mode, uint16_t& idx, Instr& ins)
  {
    switch (state_[id]) {
      case kVarS:
        mode = kModeVar;
        idx = (uint16_t)p_.nodes[id].var_index;
        break;
      case kConstS:
        mode = kModeConst;
        idx = 0;
        ins.c = p_.nodes[id].constant;
        break;
      case kAccS:
        mode = kModeAcc;
        idx = 0;
        break;
      default:
        mode = kModeSlot;
        idx = (uint16_t)slot_of_[id];
        break;
    }
  }

  void emit_generic(int64_t id, const cmn_node& nd)
  {
    int64_t a_id = nd.in0;
    int64_t b_id = nd.n_in >= 2 ? nd.in1 : nd.in0;
    materialise(a_id);
    if (nd.n_in >= 2) materialise(b_id);
    if (nd.n_in >= 2 && state_[a_id] == kConstS && state_[b_id] == kConstS) {
      // both operands constant: stage one of them in a slot
      const int s = alloc_slot();
      Instr ld = blank();
      ld.head = make_head(kOpConstToSlot, 0);
      ld.dst = (uint16_t)s;
      ld.c = p_.nodes[a_id].constant;
      emit(ld);
      Instr ins = blank();
      ins.head = make_head(kOpGeneric, (uint8_t)nd.op);
      uint8_t mb;
      uint16_t ib;
      operand(b_id, mb, ib, ins);
      ins.modes = (uint8_t)(kModeSlot | (mb << 2));
      ins.a = (uint16_t)s;
      ins.b = ib;
      consume(a_id);
      consume(b_id);
      free_slots_.push_back(s);
      ins.dst = (uint16_t)alloc_slot();
      emit(ins);
      state_[id] = kSlotS;
      slot_of_[id] = ins.dst;
      return;
    }
    Instr ins = blank();
    ins.head = make_head(kOpGeneric, (uint8_t)nd.op);
    // unary ops read no second operand: point it at the accumulator so the
    // interpreter's uniform operand fetch never indexes a slot
    uint8_t ma, mb = kModeAcc;
    uint16_t ia, ib = 0;
    operand(a_id, ma, ia, ins);
    if (nd.n_in >= 2) operand(b_id, mb, ib, ins);
    ins.modes = (uint8_t)(ma | (mb << 2));
    ins.a = ia;
    ins.b = ib;
    if (nd.op == CMN_OP_POWN) ins.b = (uint16_t)(int16_t)nd.int_exp;
    consume(a_id);
    if (nd.n_in >= 2) consume(b_id);
    ins.dst = (uint16_t)alloc_slot();
    emit(ins);
    state_[id] = kSlotS;
    slot_of_[id] = ins.dst;
  }

  Instr term_instr(const TermForm& f, uint8_t flags)
  {
    Instr ins = blank();
    uint8_t sub = (uint8_t)(flags | f.pkind | (f.has_c ? kTermHasC : 0));
    ins.head = make_head(kOpTerm, sub);
    ins.a = f.a;
    ins.b = f.b;
    ins.c = f.has_c ? f.c : 0.0;
    ++out_.n_terms;
    return ins;
  }

  // Add/Sub whose operand `t` is a deferred term: fold it into the
  // accumulator.  Returns false when the shape does not fit.
  bool try_chain(int64_t id, const cmn_node& nd)
  {
    const bool is_sub = nd.op == CMN_OP_SUB;
    const int64_t L = nd.in0, R = nd.in1;
    const bool r_term = state_[R] == kDeferred && consumer_[R] == id;
    const bool l_term = state_[L] == kDeferred && consumer_[L] == id;
    if (L == R) return false;
    int64_t base = -1, term = -1;
    uint8_t flag = 0;
    if (r_term) {
      base = L;
      term = R;
      flag = is_sub ? kTermSub : 0;
    } else if (l_term && !is_sub) {
      base = R;
      term = L;
    } else {
      return false;
    }
    // bring `base` into the accumulator
    if (state_[base] == kDeferred && consumer_[base] == id) {
      // both operands are terms: acc = base_term, then acc (+|-)= term
      spill_acc();
      emit(term_instr(form_[base], kTermInit));
      state_[base] = kNone;
    } else if (state_[base] == kAccS && acc_holder_ == base && uses_[base] == 1) {
      // running sum already in the accumulator
    } else {
      materialise(base);
      if (state_[base] == kAccS && acc_holder_ == base) {
        // still needed elsewhere: keep a copy in a slot
        spill_acc();
      }
      spill_acc();
      Instr ld = blank();
      ld.head = make_head(kOpLoadAcc, 0);
      uint8_t m;
      uint16_t ix;
      operand(base, m, ix, ld);
      ld.modes = m;
      ld.a = ix;
      emit(ld);
      consume(base);
      emit(term_instr(form_[term], flag));
      state_[term] = kNone;
      state_[id] = kAccS;
      acc_holder_ = id;
      return true;
    }
    if (state_[base] == kAccS) consume(base);
    emit(term_instr(form_[term], flag));
    state_[term] = kNone;
    state_[id] = kAccS;
    acc_holder_ = id;
    return true;
  }

  void emit_roots(int64_t id)
  {
    if (id == p_.objective_root) {
      Instr ins = blank();
      ins.head = make_head(kOpObjective, 0);
      uint8_t m;
      uint16_t ix;
      operand(id, m, ix, ins);
      ins.modes = m;
      ins.a = ix;
      emit(ins);
      consume(id);
    }
    for (const auto& c : p_.constraints) {
      if (c.root != id) continue;
      Instr ins = blank();
      ins.head = make_head(kOpCheck, (uint8_t)c.cmp);
      uint8_t m;
      uint16_t ix;
      operand(id, m, ix, ins);
      ins.modes = m;
      ins.a = ix;
      ins.c = c.rhs;  // after operand(): a constant operand is impossible here
      emit(ins);
      consume(id);
    }
  }

  void emit_all()
  {
    const int64_t n = (int64_t)p_.nodes.size();
    for (int64_t i = 0; i < n; ++i) {
      if (!p_.reach[i]) continue;
      const cmn_node& nd = p_.nodes[i];
      if (nd.op == CMN_OP_VAR) {
        state_[i] = kVarS;
      } else if (nd.op == CMN_OP_CONST) {
        state_[i] = kConstS;
      } else if (state_[i] == kDeferred || state_[i] == kAbsorbed) {
        // evaluated by its consumer
      } else if ((nd.op == CMN_OP_ADD || nd.op == CMN_OP_SUB) && try_chain(i, nd)) {
        // folded into the accumulator
      } else {
        // a generic node may read the accumulator directly; but if it
        // writes its own result while the accumulator holds a different
        // live value, nothing is lost (generic results go to slots)
        emit_generic(i, nd);
      }
      if (is_root_[i]) emit_roots(i);
    }
  }

  const HostProblem& p_;
  Program& out_;
  std::vector<int> uses_;
  std::vector<uint8_t> state_;
  std::vector<int> slot_of_;
  std::vector<TermForm> form_;
  std::vector<int64_t> consumer_;
  std::vector<uint8_t> is_root_;
  std::vector<int> free_slots_;
  int next_slot_ = 0;
  int max_slots_ = 0;
  int64_t acc_holder_ = -1;
};

}  // namespace

void compile_program(const HostProblem& p, Program& out)
{
  out = Program{};
  Compiler c(p, out);
  c.run();
}

}  // namespace cmn
