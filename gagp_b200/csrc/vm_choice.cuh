// Which VMs the programs of a grammar can need: the engine's choice of
// kernels, on the host.
#pragma once
#include <algorithm>

#include "lower.cuh"

namespace gb {

// Instructions (and constants) the lowering can emit for a row of at most
// `maxv` nodes, the appended RETURN included: a leaf or operation emits 1, a
// value if 2 (its jumps), and/or 5, and a traversal at most 36 of its own
// beside its four children, so at most 8 per node of a row holding
// traversals (36 + 4 children over 5 nodes).  A for_range emits 23 of its
// own; its body's root is a block node that emits none and is no other
// loop's body root, so at most 12 per node of a row holding loops.  A
// bounded region emits its BOUNDED_REGION and at most 13 record
// instructions beside at least five children: at most 3 per node.
// Program, block and nil nodes emit nothing, an if_stmt 2 and an assign,
// a return or a local read 1.
inline int bytecode_bound(const gagp_grammar* g, int maxv) {
  int per_node = 1;
  for (int i = 0; i < g->expression_count; ++i) {
    const int nk = g->expressions[i].node_kind;
    if (g->expressions[i].kind == EK_OPERATION)
      per_node = std::max(per_node, nk == TK_FOR_RANGE ? 12 : nk == TK_TRAVERSE ? 8 : nk == TK_REGION ? 3
                                    : nk == TK_IF ? 2
                                    : (nk == TK_AND || nk == TK_OR) ? 5 : 1);
  }
  return per_node * maxv + 2;
}

// Whether every instruction a program of `g` can emit costs one unit of
// fuel: the accumulator VM's timeout proof counts instructions.
inline bool unit_fuel(const gagp_grammar* g) {
  if (g->return_fuel != 1) return false;
  for (int r = 0; r < g->region_count; ++r)
    if (g->regions[r].fuel_profile) return false;
  for (int i = 0; i < g->expression_count; ++i)
    if (g->expressions[i].fuel != 1 || g->expressions[i].merge_fuel != 1) return false;
  return true;
}

// Whether a grammar's programs mostly need the exact VM (it sizes the VMs'
// grids): it holds traversals or bound reads, or operations that can raise a
// runtime error (modulo and division by zero, list builtins).
inline bool exact_heavy(const gagp_grammar* g) {
  if (is_statement_tag(g->slot_type)) return true;  // statement programs run on the exact VM only
  if (!unit_fuel(g)) return true;                   // so do programs with fuel charges other than 1
  for (int i = 0; i < g->expression_count; ++i) {
    const gagp_expression& e = g->expressions[i];
    if (e.kind == EK_BOUND) return true;
    if (e.kind != EK_OPERATION) continue;
    if (e.node_kind == TK_TRAVERSE) return true;
    if (e.node_kind == TK_OPERATION && accumulator_op_of(e.node_kind, e.opcode, e.operand) == A_COUNT) return true;
  }
  return false;
}

// Whether any program of a grammar can need the exact VM or the
// bounded-region kernel.  Without it those VMs are not launched and a row the
// accumulator lowering rejects is an error, so the rule asks for each of that
// lowering's reasons to reject a row the reference's compiler takes: a charge
// other than 1 or a statement (both in exact_heavy), a node it has no
// operation for (a let, a bounded region, a traversal, a bound read, an
// operation that can fail), a bytecode longer than the fuel, more than
// kMaxTemps temporaries.  The fewest nodes of a tree of need k are T(k) = 1 +
// min(2 T(k-1), 3 T(k-2)) (two children of need k-1, or an if over three of
// need k-2), T(0) = 2, T(1) = 5: a seventh temporary takes T(7) = 135 nodes.
inline bool exact_possible(const gagp_grammar* g, int fuel) {
  static_assert(kMaxTemps == 6, "the node bound is the seventh temporary's");
  const int maxv = g->max_nodes - g->fixed_nodes;
  if (exact_heavy(g) || maxv >= 135 || bytecode_bound(g, maxv) > fuel) return true;
  for (int i = 0; i < g->expression_count; ++i) {
    const gagp_expression& e = g->expressions[i];
    if (e.kind != EK_REFERENCE && !accumulator_takes(e.node_kind, e.opcode, e.operand, e.arity)) return true;
  }
  return false;
}

}  // namespace gb
