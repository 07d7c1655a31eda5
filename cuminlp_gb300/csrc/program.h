// program.h -- the fused evaluator's instruction set, shared by the host
// compiler (program.cpp) and the device interpreter (eval_core.cuh).
//
// A problem's expression DAG (model/dag.hpp:58-93 in the reference) is
// compiled once into a straight-line program over three kinds of storage:
//
//   VAR    the box's own variable intervals, staged per thread in shared
//          memory (the child box decoded from its parent in the kernel
//          prologue);
//   SLOT   a shared-memory value slot, allocated by liveness so that a
//          value occupies a slot only between its definition and last use;
//   ACC    one register-resident accumulator that carries the running sum
//          of a sum chain (sum_k c_k * x_i * x_j ...) without touching
//          shared memory.
//
// The reference evaluates every DAG node with its own kernel and a full
// HBM round trip per node (graph/builder.cuh:261-514); here a node's value
// lives in a register or in shared memory, and only the box goes in and
// the verdict comes out.  Every instruction performs exactly the rounding
// steps of the DAG nodes it stands for, in the same order, so the
// enclosures are bit-identical to node-by-node evaluation.
#pragma once

#include <cstdint>

namespace cmn {

enum OperandMode : uint8_t {
  kModeSlot = 0,
  kModeVar = 1,
  kModeAcc = 2,
  kModeConst = 3,
};

enum Opcode : uint8_t {
  // generic node: dst slot <- op(a, b)
  kOpGeneric = 0,
  // fused sum-chain term: acc <- acc (+|-) [c *] P,   P in {x_a*x_b,
  // sqr(x_a), x_a}; or acc <- [c *] P when kTermInit is set
  kOpTerm = 1,
  // slot <- acc
  kOpStoreAcc = 2,
  // acc <- operand a
  kOpLoadAcc = 3,
  // slot <- constant c (as a point interval / outward FP32 interval)
  kOpConstToSlot = 4,
  // feasibility of one constraint root: flag &= (lb <= rhs) [LE] or
  // (lb <= rhs <= ub) [EQ]; rhs in c
  kOpCheck = 5,
  // objective root: obj <- operand a
  kOpObjective = 6,
};

// node ops understood by kOpGeneric (values of cmn_op)
enum GenericOp : uint8_t {
  kGAdd = 2,
  kGSub = 3,
  kGMul = 4,
  kGDiv = 5,
  kGSqr = 6,
  kGNeg = 7,
  kGExp = 8,
  kGLog = 9,
  kGSqrt = 10,
  kGSin = 11,
  kGCos = 12,
  kGTanh = 13,
  kGPowN = 14,
  kGPow = 15,
  kGAbs = 16,
  kGMin = 17,
  kGMax = 18,
};

// kOpTerm flags (the sub-code of a term instruction)
enum TermFlags : uint8_t {
  kTermInit = 1,     // acc <- t   (start of a chain)
  kTermSub = 2,      // acc <- acc - t
  kTermHasC = 4,     // t = c * P
  kTermProd = 0,     // P = x_a * x_b      (bits 3-4)
  kTermSqr = 8,      // P = sqr(x_a)
  kTermVar = 16,     // P = x_a
  kTermPMask = 24,
};

// 16 bytes.  `head` packs the Opcode (bits 0-2) with its sub-code (bits
// 3-7: the GenericOp, the TermFlags, or the Cmp of a check).  For FP64
// programs `c` is the payload; for FP32 programs the same bytes hold the
// outward-rounded pair (clo, chi).
struct Instr {
  uint8_t head;
  uint8_t modes;  // bits 0-1 mode of a, bits 2-3 mode of b
  uint16_t dst;   // slot
  uint16_t a;     // var index / slot index
  uint16_t b;     // var index / slot index / PowN exponent (int16)
  union {
    double c;
    struct {
      float clo;
      float chi;
    } c32;
  };
};
static_assert(sizeof(Instr) == 16, "Instr layout");

// ---- sum-chain programs (Program::chain_*) ----
// One term of a chain's FP32 filter: c * x_a * x_b, c * sqr(x_a) or c * x_a.
struct ChainTerm {
  uint32_t ab;  // a in the low half, b in the high
  float c;
};

// One chain term of the FP32 passes in program order: |c| * sgn * x_a * x_b
// as an outward pair (the plane past the last variable holds [1, 1], so a
// linear term is a product too), or sqr(x_a).
struct ChainTerm32 {
  uint32_t ab;     // a in the low half, b in the high
  uint32_t flags;  // ChainTerm32Flags
  float cl, ch;    // |c| rounded outward; 1 without a coefficient
};

enum ChainTerm32Flags : uint32_t {
  kT32Neg = 0x80000000u,  // the product's sign bit
  kT32Sqr = 1u,           // sqr(x_a)
  kT32Sub = 2u,           // subtracted: the sign is folded into kT32Neg
  kT32Raw = 4u,           // x_a itself: a zero keeps its sign
  kT32Const = 8u,         // the constant [cl, ch] (signed)
};

enum ChainKind : int32_t {
  kChainObjective = 0,  // read by the objective alone: one or both bounds
  kChainGeneral = 1,    // any other reader: the two-sided interpreter
  kChainLe = 2,         // read by one <= check alone: its lower bound
};

// One sum chain and its reader.
struct ChainSeg {
  int32_t kind;
  int32_t pc0, pc1, pc2;  // chain instructions [pc0, pc1), readers [pc1, pc2)
  // the filter's terms (kChainLe, kChainObjective, eq), by sign of the coefficient and product
  // form -- [0,1) c > 0 x_a x_b, [1,2) c < 0 x_a x_b, [2,3) / [3,4) sqr,
  // [4,5) / [5,6) linear; every group padded to an even length with c = 0
  int32_t group[7];
  float c0;              // constant start of the chain
  float eps;             // FP32 error per unit of summed magnitude; 0: no filter
  float rhs_dn, rhs_up;  // the right side rounded outward
  int32_t eq;            // kChainGeneral read by one == check alone
  double rhs;
  int32_t t32, t32_end;  // the chain's terms in ChainTab::term32
  int32_t pt, pt_end;    // and in ChainTab::term_pt
};

// The chains of one program on the device: the one the objective reads
// first, then the general ones, then the <= chains, longest first.
struct ChainTab {
  const ChainSeg* seg;
  const ChainTerm* term;
  int32_t n_seg;           // 0: the program is not a set of sum chains
  int32_t pure_objective;  // the first one is kChainObjective
  int32_t points;          // points of the root box can be filtered in FP32
  // FP32 passes: every chain is kChainObjective or kChainLe and every
  // coefficient within the range of their fast arithmetic (null: not so).
  // The terms of chain q that read variable v, in program order, are
  // var32[var_off[v * n_seg + q] .. var_off[v * n_seg + q + 1]), x_v as a.
  const ChainTerm32* term32;
  const ChainTerm32* var32;
  const int32_t* var_off;
  // FP32 points: the terms in program order as c * x_a * x_b, rounded to
  // nearest, subtracted ones with -c, linear ones with the plane past the
  // last variable as x_b (null: some chain has other readers)
  const ChainTerm* term_pt;
  int32_t n_vars;
  int32_t warps32;  // warps of a tile that keep its chains' lengths balanced
  // what the choice of a path goes by: the <= chains and their terms, the
  // kChainGeneral ones and theirs
  int32_t constraints, constraint_terms;
  int32_t general, general_terms;
  int32_t products;  // terms of all chains that are products or squares
};

// A program laid out in levels (Program::level_*), on the device.
struct LevelTab {
  const Instr* prog64;
  const Instr* prog32;
  const int32_t* off;
  const int32_t* run;
  int32_t levels;  // 0: none
  int32_t slots;
};
constexpr int kLevelWarps = 8;

// Largest bound of a variable the FP32 filters take (cut32): 2^40.
constexpr double kFilterMax = 1099511627776.0;

inline constexpr uint8_t make_head(uint8_t code, uint8_t sub)
{
  return static_cast<uint8_t>(code | (sub << 3));
}

}  // namespace cmn
