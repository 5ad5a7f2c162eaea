// Exact evaluation of programs the accumulator VM cannot run: list programs
// (traversals, len, index), statement programs, lets, operations that can
// fail and grammars with fuel charges.
//
// Two parts: lower_exact_warp turns a phase row straight into register code,
// by one warp, and run_exact runs register code on the 32 cases of a tile.
// Rows that do not fit (a bounded region, or a limit below) take the
// reference bytecode (lower_program) and the per-thread interpreter
// (run_program), which also decide what is rejected.
//
// Register code.  An instruction names slots instead of a stack: the
// evaluator inputs, the grammar locals, the program's distinct constants and
// a temporary per open operand, so that the reads of inputs, binders, locals
// and constants -- more than half of the bytecode -- are operands and not
// instructions.  A traversal's step (advance, test, element, index) is one
// instruction, as are a comparison with the branch on it and a value if whose
// branches are small and cannot fail (a select; its two path costs differ, so
// it carries their difference).
//
// Fuel and errors are the reference's (cpp/src/runtime/cpu/
// execute_bytecode_cpu.cpp:152-626, the charges of
// device/phase_compile.cuh:207-895).  Every runtime failure scores the same,
// so a case fails exactly when its path's summed charges exceed the fuel or
// an operation on its path fails, in whatever order that is noticed.  Charges
// are therefore summed per straight-line stretch: word w of an instruction
// holds the charge and the bytecode instruction count from there through the
// next control instruction, and a case pays it when it arrives there by a
// jump, by falling through a control instruction or at a join.  Loops end in
// control instructions, so every loop is bounded by the fuel.
#pragma once
#include "lower.cuh"
#include "vm.cuh"

namespace gb {

// x: op | a << 8 | b << 16 | d << 24 (slots); y: jump target | slots; z: select
// operands or immediate; w: charge | instructions << 16 (see above).
enum : uint32_t {
  X_MOVE = 0, X_IMM, X_NEG, X_NOT, X_ABS, X_LEN, X_INDEX,
  X_ADD, X_SUB, X_MUL, X_MOD, X_LT, X_LE, X_GT, X_GE, X_EQ, X_NE,  // the order of OP_ADD.., OP_LT..
  X_MIN, X_MAX, X_IDIV0, X_IMOD0, X_TDIV0, X_TMOD0,
  X_SEL_LT, X_SEL_LE, X_SEL_GT, X_SEL_GE, X_SEL_EQ, X_SEL_NE,      // d = (a ? b) ? y0 : y1, z: the true path's extra charge
  X_BEGIN, X_BEGIN_REVERSE, X_ELEMENT,
  X_CONTROL,                                                       // from here on: control instructions
  X_JLT = X_CONTROL, X_JLE, X_JGT, X_JGE, X_JEQ, X_JNE, X_JT, X_JF, X_JMP, X_RET, X_FAIL,
  X_TEST, X_NEXT, X_NEXT_REVERSE, X_FOR, X_FOR_NEXT, X_COUNT
};

constexpr int kExactSlots = 32;    // slots of a program: 8 KB of shared memory per warp
constexpr int kExactConsts = 8;    // of which at most these hold constants
constexpr int kExactWords = 384;   // instructions of a program
constexpr int kExactDepth = 48;    // nesting of a row (below every capacity of the reference's compiler)
constexpr int kSelectNodes = 8;    // nodes of both branches of a select
constexpr int8_t kNoType = GAGP_TAG_INVALID;

// Per-warp shared memory of lower_exact_warp.
struct ExactScratch {
  uint32_t fuel[kMaxLowerNodes + 1];   // charges of the nodes before this one
  uint32_t cw[kExactWords];            // a word's charge | instructions << 16 | control << 31
  int16_t end[kMaxLowerNodes];         // one past the subtree
  int16_t words[kMaxLowerNodes + 1];   // words of the nodes before this one
  int16_t start[kMaxLowerNodes];       // open slots; not-flat nodes so far; then the first word's offset from the parent's
  int16_t at[kMaxLowerNodes];          // a traversal's or a let's binder numbers; then the subtree's first word
  uint8_t pos[kMaxLowerNodes];         // temporaries the parent holds while the node runs
  uint8_t slot[kMaxLowerNodes];        // temporaries all ancestors hold
  uint8_t par[kMaxLowerNodes], kind[kMaxLowerNodes], flags[kMaxLowerNodes], mark[kMaxLowerNodes];
  // by class: an operation's register operation, an input's or a grammar
  // local's slot, a bound read's binder node, a constant's slot rank (0xff:
  // an immediate), the slot an assignment or a loop stores to
  uint8_t aux[kMaxLowerNodes];
  int8_t type[kMaxLowerNodes];         // completion type (an if's and a let's: type_of)
};

// Node classes.
enum : uint8_t {
  N_CONST = 0, N_SLOT, N_BOUND, N_OP1, N_OP2, N_IF, N_AND, N_OR, N_LET, N_TRAVERSE, N_SEQUENCE, N_NIL, N_ASSIGN, N_RETURN,
  N_FOR, N_BAD
};
// Node flags: the child's number; a comparison its if's branch performs; an
// if that is a select; a node inside a select's branches; a comparison; which
// of a traversal's binders a bound read names (bits 6-7).
enum : uint8_t { NF_ORD = 3, NF_FUSED = 4, NF_SELECT = 8, NF_INSIDE = 16, NF_COMPARE = 32 };
// Marks: the value goes straight into a slot of the parent; a leaf read where
// it is used (no word, no temporary); a traversal body that is the
// traversal's own state (nothing to do).
enum : uint8_t { NM_DIRECTED = 1, NM_ALIAS = 2, NM_IDLE = 4 };

// Register operation of an operation node; X_COUNT: none.
__device__ __forceinline__ uint32_t exact_op_of(int opcode, int operand, int arity) {
  if (opcode == OP_CALL_BUILTIN) {
    switch (operand) {
      case B_ABS: return arity == 1 ? X_ABS : X_COUNT;
      case B_LEN: return arity == 1 ? X_LEN : X_COUNT;
      case B_INDEX: return arity == 2 ? X_INDEX : X_COUNT;
      case B_MIN: return arity == 2 ? X_MIN : X_COUNT;
      case B_MAX: return arity == 2 ? X_MAX : X_COUNT;
      case B_IDIV0: return arity == 2 ? X_IDIV0 : X_COUNT;
      case B_IMOD0: return arity == 2 ? X_IMOD0 : X_COUNT;
      case B_TRUNC_DIV0: return arity == 2 ? X_TDIV0 : X_COUNT;
      case B_TRUNC_MOD0: return arity == 2 ? X_TMOD0 : X_COUNT;
      default: return X_COUNT;
    }
  }
  if (opcode == OP_NEG) return arity == 1 ? X_NEG : X_COUNT;
  if (opcode == OP_NOT) return arity == 1 ? X_NOT : X_COUNT;
  if (arity != 2) return X_COUNT;
  if (opcode == OP_MOD) return X_MOD;
  if (opcode >= OP_ADD && opcode <= OP_MUL) return X_ADD + uint32_t(opcode - OP_ADD);
  if (opcode >= OP_LT && opcode <= OP_NE) return X_LT + uint32_t(opcode - OP_LT);
  return X_COUNT;
}

// The warp's sum of `v` over the lanes before this one, and the total.
__device__ __forceinline__ uint32_t warp_prefix(uint32_t v, uint32_t* total) {
  const int lane = threadIdx.x & 31;
  uint32_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += t;
  }
  *total = __shfl_sync(kFull, incl, 31);
  return incl - v;
}

// Register code of a row, by one warp; the instruction count (the same on
// every lane), or -1 when the row takes the reference bytecode instead.
// words: [0] instructions | constants << 16, first constant slot; the
// instructions follow, and one more word may be read past the last.
//
// What bounds it: latency (a chain of shared-memory passes over the nodes, a
// pass per question; about 40k cycles beside a full round's other warps).
// The bytecode lowering walks the tree on one lane instead: 86 us a range of
// 1024 list-program children against 47 us here.  Every node's words,
// temporaries and charges follow from sums along its path from the root and
// over the nodes before it, as in lower_accumulator_emit, so the lanes share
// the nodes; what several passes ask of a node (its operation, binder, type)
// is kept in shared memory, which took the walk from 143 to 47 us.
__device__ __noinline__ int lower_exact_warp(const SearchDesc& s, const uint64_t* node, int n, const int64_t* cval,
                                             int nc, uint4* words, int word_cap, int64_t* consts, ExactScratch& m) {
  const int lane = threadIdx.x & 31;
  if (n <= 0 || n > kMaxLowerNodes) return -1;
  const bool statements = is_statement_tag(s.slot_type);
  const int n_inputs = s.local_count;
  if (n_inputs > kExactSlots || s.return_fuel > 0xffu) return -1;
  bool bad = false;
  int named = 0;
  // ---- classes, charges, open slots
  {
    const bool unit = s.unit_fuel;
    uint32_t open = 1, fuel = 0, seen = 0;
    for (int base = 0; base < n; base += 32) {
      const int i = base + lane;
      uint32_t charge = 0;
      int arity = 1;
      bool is_const = false;
      if (i < n) {
        const uint64_t w = node[i];
        const int o = w_origin(w);
        arity = w_arity(w);
        uint8_t kind = N_BAD, aux = 0, flags = 0;
        int8_t type = kNoType;
        if (o < s.n_ex) {
          // kind, node kind, arity and type, then the opcode (the table is 256-byte aligned)
          static_assert(sizeof(ExprInfo) % 8 == 0, "read in 8-byte words");
          const int2 raw = __ldg(reinterpret_cast<const int2*>(&s.info[o]));
          const int nk = int8_t(raw.x >> 8), opcode = int16_t(raw.y), operand = __ldg(&s.info[o].operand);
          type = int8_t(raw.x >> 24);
          charge = 1;
          if (!unit) {
            charge = s.ex[o].fuel;
            bad |= charge > 0xffu || s.ex[o].merge_fuel > 0xffu;
          }
          int want = -1;
          const int stored = operand < 0 ? -1 - operand : n_inputs + operand;  // an assignment's or a loop's variable
          switch (nk) {
            case TK_CONSTANT: kind = N_CONST; want = 0; type = GAGP_TAG_INT; is_const = true; break;
            case TK_LOCAL:
              kind = N_SLOT; want = 0;
              bad |= operand < 0 || operand >= n_inputs;
              if (operand >= 0 && operand < n_inputs) { aux = uint8_t(operand); type = int8_t(s.local_types[operand]); }
              break;
            case TK_BOUND: kind = N_BOUND; want = 0; aux = uint8_t(operand); bad |= operand < 0 || operand >= kLowerBinders; break;
            case TK_VAR:
              kind = N_SLOT; want = 0;
              bad |= operand < 0 || operand >= kNamedLocals || type == GAGP_TAG_INVALID || is_statement_tag(type);
              aux = uint8_t(stored);
              named = max(named, operand + 1);
              break;
            case TK_OPERATION: {
              const uint32_t op = exact_op_of(opcode, operand, arity);
              kind = op == X_COUNT ? N_BAD : arity == 1 ? N_OP1 : N_OP2;
              want = arity;
              aux = uint8_t(op);
              if (op >= X_LT && op <= X_NE) flags = NF_COMPARE;
              break;
            }
            case TK_IF: kind = N_IF; want = 3; break;
            case TK_AND: kind = N_AND; want = 2; type = GAGP_TAG_BOOL; break;
            case TK_OR: kind = N_OR; want = 2; type = GAGP_TAG_BOOL; break;
            case TK_LET:
              kind = N_LET; want = 2;
              bad |= operand < 0 || operand >= kLowerBinders;
              m.at[i] = int16_t(operand);
              break;
            case TK_TRAVERSE:
              kind = N_TRAVERSE; want = 4;
              if (operand < 0 || operand >= s.n_regions) bad = true;
              else {
                const RegionInfo& r = s.regions[operand];
                bad |= (r.traversal != 1 && r.traversal != 2) || r.ranged || r.arity != 4;
                for (int k = 0; k < 3; ++k) bad |= r.binders[k] < 0 || r.binders[k] >= kLowerBinders;
                for (int k = 4; k < 26 && r.fuel_profile; ++k) bad |= r.event_cost[k] > 0xffu;
                m.at[i] = int16_t(r.binders[0] | r.binders[1] << 4 | r.binders[2] << 8);
                type = r.result_type;
              }
              break;
            case TK_PROGRAM: kind = N_SEQUENCE; want = 1; break;
            case TK_BLOCK: kind = N_SEQUENCE; want = 2; break;
            case TK_NIL: kind = N_NIL; want = 0; break;
            case TK_ASSIGN: case TK_FOR_RANGE:
              kind = nk == TK_ASSIGN ? N_ASSIGN : N_FOR;
              want = nk == TK_ASSIGN ? 1 : 2;
              bad |= operand >= kNamedLocals || (operand < 0 && -1 - operand >= n_inputs);
              aux = uint8_t(stored);
              named = max(named, operand + 1);
              break;
            case TK_RETURN: kind = N_RETURN; want = 1; break;
            default: break;
          }
          bad |= arity != want || int8_t(raw.x >> 16) != arity;
        }
        bad |= kind == N_BAD;
        m.kind[i] = kind;
        m.aux[i] = aux;
        m.flags[i] = flags;
        m.type[i] = type;
      }
      uint32_t total;
      const uint32_t before = warp_prefix(i < n ? uint32_t(arity - 1) : 0u, &total);
      if (i < n) m.start[i] = int16_t(open + before);
      open += total;
      const uint32_t fuel_before = warp_prefix(charge, &total);
      if (i < n) m.fuel[i] = fuel + fuel_before;
      fuel += total;
      seen += __popc(__ballot_sync(kFull, is_const));
    }
    if (lane == 0) m.fuel[n] = fuel;
    bad |= open != 0 || seen > uint32_t(nc);
  }
  named = __reduce_max_sync(kFull, named);
  if (__any_sync(kFull, bad)) return -1;
  __syncwarp();
  const int base_slot = n_inputs + named;
  if (base_slot > kExactSlots) return -1;
  // ---- constants: the first 32 by their values, the first kExactConsts
  // distinct values in slots; a constant node's rank, then its slot (0xff: an
  // immediate)
  int const_count = 0;
  uint32_t const_rank = 0xff;  // lane k: slot rank of constant k
  {
    const int64_t v = lane < nc ? cval[lane] : 0;
    const unsigned live = __ballot_sync(kFull, lane < nc);
    if (lane < nc) {
      const int first = __ffs(__match_any_sync(live, v)) - 1;
      const unsigned firsts = __ballot_sync(live, first == lane);
      const_rank = uint32_t(__popc(firsts & ((1u << first) - 1)));
      if (first == lane && const_rank < kExactConsts) consts[const_rank] = v;
      const_count = min(__popc(firsts), kExactConsts);
    }
    const_count = __shfl_sync(kFull, const_count, 0);
  }
  // ---- subtree ends (as in lower_accumulator_emit) and parents
  for (int base = 0; base < n; base += 32) {
    const int i = base + lane;
    const int r = i < n ? m.start[i] : 0;
    int e = n;
    bool found = i >= n;
    for (int cb = base; cb < n && __any_sync(kFull, !found); cb += 32) {
      const int j = cb + lane;
      const int open = j < n ? m.start[j] : 0x7fffffff;
      for (int q = 0; q < 32; ++q) {
        const int rq = __shfl_sync(kFull, r, q);
        const unsigned hit = __ballot_sync(kFull, j > base + q && open < rq);
        if (lane == q && !found && hit) {
          e = cb + __ffs(hit) - 1;
          found = true;
        }
      }
    }
    if (i < n) m.end[i] = int16_t(e);
  }
  __syncwarp();
  if (m.end[0] != n) return -1;
  {
    int rank = 0;
    for (int base = 0; base < n; base += 32) {
      const int i = base + lane;
      const bool is_const = i < n && m.kind[i] == N_CONST;
      const unsigned mask = __ballot_sync(kFull, is_const);
      const int k = rank + __popc(mask & ((1u << lane) - 1));
      const uint32_t slot = __shfl_sync(kFull, const_rank, k & 31);
      if (i < n) {
        if (is_const) m.aux[i] = k < 32 && slot < kExactConsts ? uint8_t(slot) : uint8_t(0xff);
        const int a = w_arity(node[i]);
        for (int x = 0, c = i + 1; x < a; ++x) {
          if (c >= n) { bad = true; break; }
          m.par[c] = uint8_t(i);
          m.flags[c] = uint8_t((m.flags[c] & ~NF_ORD) | x);
          c = m.end[c];
        }
      }
      rank += __popc(mask);
    }
  }
  if (__any_sync(kFull, bad)) return -1;
  __syncwarp();
  auto ex_of = [&](int i) -> const gagp_expression& { return s.ex[w_origin(node[i])]; };
  auto child = [&](int i, int x) {
    int c = i + 1;
    for (; x > 0; --x) c = m.end[c];
    return c;
  };
  // completion type of node i (lower_code's `completed`): statements have
  // the statement tag
  auto type_of = [&](int i) -> int {
    while (m.kind[i] == N_IF || m.kind[i] == N_LET) i = child(i, 1);
    return m.kind[i] >= N_SEQUENCE ? kStatementTag : int(m.type[i]);
  };
  // ---- bound reads: the nearest traversal body (element, index or state)
  // or let body around the node that binds its number
  for (int i = lane; i < n; i += 32) {
    if (m.kind[i] != N_BOUND) continue;
    const int b = m.aux[i];
    int binder = -1, which = 0;
    for (int x = i; x > 0 && binder < 0; x = m.par[x]) {
      const int p = m.par[x], ord = m.flags[x] & NF_ORD;
      if (m.kind[p] == N_LET && ord == 1 && m.at[p] == b) {
        binder = p;
      } else if (m.kind[p] == N_TRAVERSE && ord == 3) {
        for (int k = 2; k >= 0 && binder < 0; --k)
          if ((m.at[p] >> (4 * k) & 15) == b) { binder = p; which = k; }
      }
    }
    bad |= binder < 0;
    m.aux[i] = uint8_t(max(binder, 0));
    m.flags[i] |= uint8_t(which << 6);
  }
  if (__any_sync(kFull, bad)) return -1;
  __syncwarp();
  // their types: the traversal's binding, or the let's value (a let's value
  // may itself be read through another let, so outer ones come first)
  for (int i = lane; i < n; i += 32) {
    if (m.kind[i] != N_BOUND) continue;
    int x = i, t = GAGP_TAG_INVALID;
    for (int guard = 0; guard < kExactDepth; ++guard) {
      const int p = m.aux[x];
      if (m.kind[p] == N_TRAVERSE) {
        t = s.regions[ex_of(p).operand].binding_types[m.flags[x] >> 6];
        break;
      }
      int y = p + 1;
      while (m.kind[y] == N_IF || m.kind[y] == N_LET) y = child(y, 1);
      if (m.kind[y] != N_BOUND) { t = type_of(y); break; }
      x = y;
    }
    bad |= t == GAGP_TAG_INVALID || (m.type[i] != GAGP_TAG_INVALID && m.type[i] != t);
    m.type[i] = int8_t(t);
  }
  __syncwarp();
  // ---- what the compiler checks, and which subtrees are flat
  // (loads and operations that cannot fail: a select may run both branches)
  {
    uint32_t not_flat = 0;
    for (int base = 0; base < n; base += 32) {
      const int i = base + lane;
      bool flat = true;
      if (i < n) {
        const uint8_t kind = m.kind[i];
        const uint32_t op = m.aux[i];
        flat = kind <= N_BOUND || ((kind == N_OP1 || kind == N_OP2) && op != X_MOD && op != X_INDEX);
        switch (kind) {
          case N_OP1: case N_OP2: {
            // operands of other types fail at run time: run_program's checks
            const int t = type_of(i + 1);
            if (op == X_LEN || op == X_INDEX) bad |= t != GAGP_TAG_INTLIST;
            else if (op == X_NOT) bad |= t != GAGP_TAG_BOOL;
            else if (op == X_EQ || op == X_NE) bad |= t != GAGP_TAG_INT && t != GAGP_TAG_BOOL;
            else bad |= t != GAGP_TAG_INT;
            if (kind == N_OP2)
              bad |= type_of(child(i, 1)) != (op == X_EQ || op == X_NE ? t : int(GAGP_TAG_INT));
            break;
          }
          case N_IF:
            bad |= type_of(i + 1) != GAGP_TAG_BOOL || int8_t(type_of(child(i, 1))) != int8_t(type_of(child(i, 2)));
            break;
          case N_AND: case N_OR:
            bad |= type_of(i + 1) != GAGP_TAG_BOOL || type_of(child(i, 1)) != GAGP_TAG_BOOL;
            break;
          case N_LET:
            bad |= is_statement_tag(type_of(i + 1)) ||
                   (m.type[i] != GAGP_TAG_INVALID && m.type[i] != type_of(child(i, 1)));
            break;
          case N_TRAVERSE: {
            const RegionInfo& r = s.regions[ex_of(i).operand];
            for (int x = 0, c = i + 1; x < 4; ++x, c = m.end[c]) bad |= type_of(c) != r.operand_types[x];
            break;
          }
          case N_SEQUENCE:
            for (int x = 0, c = i + 1; x < int(w_arity(node[i])); ++x, c = m.end[c]) bad |= !is_statement_tag(type_of(c));
            break;
          case N_ASSIGN: case N_RETURN: {
            const int t = type_of(i + 1);
            bad |= t != m.type[i] || is_statement_tag(t);
            break;
          }
          case N_FOR:
            bad |= is_statement_tag(type_of(i + 1)) || !is_statement_tag(type_of(child(i, 1)));
            break;
          default: break;
        }
        bad |= kind >= N_SEQUENCE && !statements;  // statements only among statements
      }
      uint32_t total;
      const uint32_t before = warp_prefix(i < n && !flat, &total);
      if (i < n) m.start[i] = int16_t(not_flat + before + uint32_t(!flat));  // through node i
      not_flat += total;
    }
    bad |= type_of(0) != s.slot_type && !(statements && is_statement_tag(type_of(0)));
  }
  if (__any_sync(kFull, bad)) return -1;
  if (statements) {
    bool ok = false;
    if (lane == 0) ok = row_locals_defined(s, node, n);
    if (!__shfl_sync(kFull, ok, 0)) return -1;
  }
  __syncwarp();
  // ---- fused comparisons and selects
  for (int i = lane; i < n; i += 32) {
    if (m.kind[i] != N_IF) continue;
    const int c0 = i + 1, c1 = m.end[c0];
    if (!(m.flags[c0] & NF_COMPARE)) continue;
    const bool flat = m.start[m.end[i] - 1] == m.start[c1 - 1];
    const bool select = flat && m.end[i] - c1 <= kSelectNodes && !is_statement_tag(type_of(c1));
    m.flags[c0] |= NF_FUSED;
    if (select) {
      m.flags[i] |= NF_SELECT;
      for (int j = c1; j < m.end[i]; ++j) m.flags[j] |= NF_INSIDE;
    }
  }
  __syncwarp();
  auto alias = [&](int i) -> bool { return m.mark[i] & NM_ALIAS; };
  // ---- words
  uint32_t total_words = 0;
  for (int base = 0; base < n; base += 32) {
    const int i = base + lane;
    uint32_t own = 0;
    if (i < n) {
      const uint8_t kind = m.kind[i], flags = m.flags[i];
      const int p = m.par[i], ord = flags & NF_ORD;
      const uint8_t above = i ? m.kind[p] : uint8_t(N_SEQUENCE);
      const bool directed = above == N_ASSIGN || above == N_LET || (above == N_IF && ord > 0 && !(m.flags[p] & NF_SELECT)) ||
                            ((above == N_AND || above == N_OR) && ord == 1) || (above == N_TRAVERSE && ord >= 2) ||
                            (above == N_FOR && ord == 0);
      const bool leaf_read = !directed && (kind == N_SLOT || kind == N_BOUND || (kind == N_CONST && m.aux[i] != 0xff));
      const bool idle = kind == N_BOUND && above == N_TRAVERSE && ord == 3 && m.aux[i] == p && (flags >> 6) == 2;
      m.mark[i] = uint8_t((directed ? NM_DIRECTED : 0) | (leaf_read ? NM_ALIAS : 0) | (idle ? NM_IDLE : 0));
      switch (kind) {
        case N_CONST: case N_SLOT: case N_BOUND: own = !leaf_read && !idle; break;
        case N_OP1: case N_OP2: own = !(flags & NF_FUSED); break;
        case N_IF: own = flags & NF_SELECT ? 1 : 2; break;
        case N_AND: case N_OR: own = 3; break;
        case N_TRAVERSE: own = 4 + directed; break;
        case N_RETURN: own = 1; break;
        case N_FOR: own = 2; break;
        default: break;
      }
    }
    uint32_t total;
    const uint32_t before = warp_prefix(own, &total);
    if (i < n) m.words[i] = int16_t(min(total_words + before, 32767u));
    total_words += total;
  }
  if (lane == 0) m.words[n] = int16_t(min(total_words, 32767u));
  const int count = int(total_words) + 1;  // and the appended RETURN, or the end of a statement program
  if (count > kExactWords || count + 2 > word_cap) return -1;
  for (int k = lane; k < count; k += 32) m.cw[k] = 0;
  __syncwarp();
  auto size = [&](int i) { return m.words[m.end[i]] - m.words[i]; };
  // ---- first words and temporaries: offsets from the parent, then sums
  // along the path from the root
  for (int i = lane; i < n; i += 32) {
    if (i == 0) { m.start[0] = 0; m.pos[0] = 0; }
    const int a = w_arity(node[i]);
    const uint8_t kind = m.kind[i];
    const bool select = m.flags[i] & NF_SELECT;
    int at = 0, held = kind == N_TRAVERSE ? 5 : 0;
    for (int x = 0, c = i + 1; x < a; ++x, c = m.end[c]) {
      if (select && x == 1) {
        // the comparison's operands stay while the branches run
        const int l = i + 2, r = m.end[l];
        held = int(!alias(l)) + int(!alias(r));
      }
      m.start[c] = int16_t(at);
      m.pos[c] = uint8_t(held);
      at += size(c);
      switch (kind) {
        case N_OP2: held += x == 0 && !alias(c); break;
        case N_IF:
          if (select) held += x == 1 && !alias(c);
          else at += x < 2;
          break;
        case N_AND: case N_OR: at += x == 0; break;
        case N_LET: held = 1; break;
        case N_TRAVERSE:
          if (x < 2) held += !alias(c);
          at += x == 1 ? 1 : x == 2 ? 2 : 0;
          break;
        case N_FOR: held = 2; at += x == 0; break;
        default: break;
      }
    }
  }
  __syncwarp();
  int top = 0;  // slots in use
  for (int i = lane; i < n; i += 32) {
    int at = 0, held = 0, depth = 0;
    for (int x = i; x > 0; x = m.par[x]) {
      at += m.start[x];
      held += m.pos[x];
      ++depth;
    }
    bad |= depth >= kExactDepth;
    m.at[i] = int16_t(at);
    m.slot[i] = uint8_t(min(held, 255));
    int own = 1;
    if (m.kind[i] == N_TRAVERSE) own = 5 + int(!alias(i + 1)) + int(!alias(m.end[i + 1]));
    else if (m.kind[i] == N_FOR) own = 2;
    top = max(top, held + own);
  }
  const int const_base = base_slot + __reduce_max_sync(kFull, top);
  if (const_base + const_count > kExactSlots || __any_sync(kFull, bad)) return -1;
  __syncwarp();
  // ---- every node writes its words
  uint4* out = words + 1;
  auto fuel_of = [&](int i) -> uint32_t { return m.fuel[i + 1] - m.fuel[i]; };
  auto leaf_slot = [&](int i) -> uint32_t {
    const uint8_t kind = m.kind[i];
    const int aux = m.aux[i];
    if (kind == N_CONST) return uint32_t(const_base + aux);
    if (kind == N_SLOT) return uint32_t(aux);
    const int which = m.flags[i] >> 6;  // of a traversal: 0 element, 1 index, 2 state
    return uint32_t(base_slot + m.slot[aux] + (m.kind[aux] == N_LET || which == 2 ? 0 : 3 + which));
  };
  auto operand = [&](int i) -> uint32_t { return alias(i) ? leaf_slot(i) : uint32_t(base_slot + m.slot[i]); };
  auto leaf_cost = [&](int i) -> uint32_t { return alias(i) ? fuel_of(i) | 1u << 16 : 0u; };
  // the slot node i's value goes to
  auto target_slot = [&](int i) -> uint32_t {
    int x = i;
    while (x > 0) {
      const int p = m.par[x], ord = m.flags[x] & NF_ORD;
      const uint8_t kind = m.kind[p];
      if (kind == N_ASSIGN) return m.aux[p];
      if (kind == N_LET && ord == 0) return uint32_t(base_slot + m.slot[p]);
      if (kind == N_TRAVERSE && ord >= 2) return uint32_t(base_slot + m.slot[p]);
      if (kind == N_FOR && ord == 0) return uint32_t(base_slot + m.slot[p]);
      if (kind == N_LET || (kind == N_IF && ord > 0 && !(m.flags[p] & NF_SELECT)) ||
          ((kind == N_AND || kind == N_OR) && ord == 1)) {
        x = p;
        continue;
      }
      break;
    }
    return uint32_t(base_slot + m.slot[x]);
  };
  // the store of node i's value by an assignment or a let: it runs exactly
  // when the node's own control or last word does
  auto store_cost = [&](int i) -> uint32_t {
    for (int x = i; x > 0;) {
      const int p = m.par[x];
      if (m.kind[p] == N_ASSIGN) return fuel_of(p) | 1u << 16;
      if (m.kind[p] != N_LET) return 0;
      if ((m.flags[x] & NF_ORD) == 0) return fuel_of(p) | 1u << 16;
      x = p;
    }
    return 0;
  };
  auto put = [&](int k, uint32_t op, uint32_t a, uint32_t b, uint32_t d, uint32_t y, uint32_t z, uint32_t cost) {
    out[k] = make_uint4(op | a << 8 | b << 16 | d << 24, y, z, 0);
    atomicAdd(&m.cw[k], cost + (op >= X_CONTROL ? 1u << 31 : 0u));
  };
  int rank = 0;
  for (int base = 0; base < n; base += 32) {
    const int i = base + lane;
    const bool live = i < n;
    const uint8_t kind = live ? m.kind[i] : uint8_t(N_NIL);
    const unsigned const_mask = __ballot_sync(kFull, kind == N_CONST);
    const int row_const = rank + __popc(const_mask & ((1u << lane) - 1));
    rank += __popc(const_mask);
    if (!live) continue;
    const int at = m.at[i];
    const bool inside = m.flags[i] & NF_INSIDE;
    const uint32_t own = inside ? 0u : fuel_of(i) | 1u << 16;
    switch (kind) {
      case N_CONST:
        if (alias(i)) break;
        if (m.aux[i] != 0xff) {
          put(at, X_MOVE, leaf_slot(i), 0, target_slot(i), 0, 0, own + store_cost(i));
        } else {
          const uint64_t v = uint64_t(cval[row_const]);
          put(at, X_IMM, 0, 0, target_slot(i), uint32_t(v), uint32_t(v >> 32), own + store_cost(i));
        }
        break;
      case N_SLOT: case N_BOUND:
        if (!(m.mark[i] & (NM_ALIAS | NM_IDLE))) put(at, X_MOVE, leaf_slot(i), 0, target_slot(i), 0, 0, own + store_cost(i));
        break;
      case N_OP1: {
        const int c = i + 1;
        put(at + size(c), m.aux[i], operand(c), 0, target_slot(i), 0, 0,
            own + (inside ? 0u : leaf_cost(c)) + store_cost(i));
        break;
      }
      case N_OP2: {
        if (m.flags[i] & NF_FUSED) break;
        const int c = i + 1, d = m.end[c];
        put(at + size(c) + size(d), m.aux[i], operand(c), operand(d), target_slot(i), 0, 0,
            own + (inside ? 0u : leaf_cost(c) + leaf_cost(d)) + store_cost(i));
        break;
      }
      case N_IF: {
        const int c0 = i + 1, c1 = m.end[c0], c2 = m.end[c1];
        const uint32_t merge_fuel = s.unit_fuel ? 1u : ex_of(i).merge_fuel;
        uint32_t a, b = 0, cost = own + store_cost(i), compare = X_COUNT;
        if (m.flags[c0] & NF_FUSED) {
          const int l = c0 + 1, r = m.end[l];
          a = operand(l);
          b = operand(r);
          cost += (fuel_of(c0) | 1u << 16) + leaf_cost(l) + leaf_cost(r);
          compare = m.aux[c0] - X_LT;
        } else {
          a = operand(c0);
          cost += leaf_cost(c0);
        }
        if (m.flags[i] & NF_SELECT) {
          // both paths' charges: the cheaper one with the straight line, the
          // difference by the path taken
          const int yes = int(m.fuel[c2] - m.fuel[c1] + merge_fuel), no = int(m.fuel[m.end[i]] - m.fuel[c2]);
          const int yes_n = c2 - c1 + 1, no_n = m.end[i] - c2;
          put(at + size(i) - 1, X_SEL_LT + compare, a, b, target_slot(i), operand(c1) | operand(c2) << 8,
              uint32_t(uint16_t(int16_t(yes - no))) | uint32_t(uint16_t(int16_t(yes_n - no_n))) << 16,
              cost + uint32_t(min(yes, no)) + (uint32_t(no_n) << 16));
          break;
        }
        // the branch not taken when the condition holds: LT/LE/GT/GE/EQ/NE inverted
        const uint32_t jump = compare == X_COUNT ? uint32_t(X_JF)
                              : compare < 4      ? X_JLT + (3 - compare)
                                                 : X_JLT + (9 - compare);
        put(at + size(c0), jump, a, b, 0, uint32_t(m.at[c2]), 0, cost);
        put(m.at[c2] - 1, X_JMP, 0, 0, 0, uint32_t(at + size(i)), 0, merge_fuel | 1u << 16);
        break;
      }
      case N_AND: case N_OR: {
        const int c0 = i + 1, last = at + size(i) - 1;
        put(at + size(c0), kind == N_AND ? X_JF : X_JT, operand(c0), 0, 0, uint32_t(last), 0,
            own + leaf_cost(c0) + store_cost(i));
        put(last - 1, X_JMP, 0, 0, 0, uint32_t(last + 1), 0, 3 * fuel_of(i) + (3u << 16));
        put(last, X_IMM, 0, 0, target_slot(i), kind == N_OR, 0, fuel_of(i) | 1u << 16);
        break;
      }
      case N_TRAVERSE: {
        const RegionInfo& r = s.regions[ex_of(i).operand];
        const bool reverse = r.traversal == 2;
        // an event's charge and instructions (lower_code's walk_after)
        auto event = [&](int which, uint32_t instructions) -> uint32_t {
          return (r.fuel_profile ? r.event_cost[which] : instructions) + (instructions << 16);
        };
        const uint32_t q = uint32_t(base_slot + m.slot[i]);  // state, cursor, limit, element, index
        const int c0 = i + 1, c1 = m.end[c0], c3 = m.end[m.end[c1]];
        const uint32_t views = operand(c0) << 16 | operand(c1) << 24;
        const int next = m.at[c3] + size(c3);
        // the result's read happens once, when the traversal completes: paid here
        put(at + size(c0) + size(c1), reverse ? X_BEGIN_REVERSE : X_BEGIN, operand(c0), 0, q + 2, 0, 0,
            leaf_cost(c0) + leaf_cost(c1) + event(4, 1) + event(5, 1) + event(8, 3) + event(11, 3) + event(14, 2) +
                event(15, 2) + event(25, 1) + store_cost(i));
        put(m.at[c3] - 2, X_TEST, q + 2, 0, 0, uint32_t(next + 1), 0, event(16, 1) + event(17, reverse ? 4 : 2) + event(18, 4));
        put(m.at[c3] - 1, X_ELEMENT, 0, q + 1, q + 3, views, 0, 0);
        // paid on entry to the body, by the first pass and by every next one
        atomicAdd(&m.cw[m.at[c3]], event(19, 3) + event(20, 1) + event(21, 4));
        put(next, reverse ? X_NEXT_REVERSE : X_NEXT, q + 1, q + 2, q + 3, uint32_t(m.at[c3]) | views, 0,
            event(22, 1) + event(23, 4) + event(24, 1) + event(18, 4) + (m.mark[c3] & NM_IDLE ? fuel_of(c3) | 1u << 16 : 0u));
        if (m.mark[i] & NM_DIRECTED) put(next + 1, X_MOVE, q, 0, target_slot(i), 0, 0, 0);
        break;
      }
      case N_RETURN:
        put(at + size(i + 1), X_RET, operand(i + 1), 0, 0, 0, 0, own + leaf_cost(i + 1));
        break;
      case N_FOR: {
        // lower_code's template, every instruction charged 1
        const uint32_t q = uint32_t(base_slot + m.slot[i]);  // bound, counter
        const int c1 = m.end[i + 1], next = m.at[c1] + size(c1);
        const uint32_t user = uint32_t(m.aux[i]) << 16;
        put(m.at[c1] - 1, X_FOR, q, 0, q + 1, uint32_t(next + 1) | user, 0, 14 + (14u << 16));
        atomicAdd(&m.cw[m.at[c1]], 2 + (2u << 16));
        put(next, X_FOR_NEXT, q + 1, q, 0, uint32_t(m.at[c1]) | user, 0, 9 + (9u << 16));
        break;
      }
      default: break;
    }
  }
  if (lane == 0) {
    if (statements) put(count - 1, X_FAIL, 0, 0, 0, 0, 0, 0);
    else put(count - 1, X_RET, operand(0), 0, 0, 0, 0, (s.return_fuel | 1u << 16) + leaf_cost(0));
    words[0] = make_uint4(uint32_t(count) | uint32_t(const_count) << 16, uint32_t(const_base), 0, 0);
  }
  __syncwarp();
  // ---- charges from each word through the next control word
  uint32_t carry_cost = 0, carry_count = 0;
  for (int base = (count - 1) & ~31; base >= 0; base -= 32) {
    const int j = base + lane;
    const uint32_t c = j < count ? m.cw[j] : 1u << 31;
    uint32_t cost = c & 0xffffu, instructions = (c >> 16) & 0x7fffu;
    bool stop = c >> 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t c2 = __shfl_down_sync(kFull, cost, o), n2 = __shfl_down_sync(kFull, instructions, o);
      const bool stop2 = __shfl_down_sync(kFull, int(stop), o);
      if (lane + o < 32 && !stop) {
        cost += c2;
        instructions += n2;
        stop = stop2;
      }
    }
    if (!stop) {
      cost += carry_cost;
      instructions += carry_count;
    }
    carry_cost = __shfl_sync(kFull, cost, 0);
    carry_count = __shfl_sync(kFull, instructions, 0);
    bad |= j < count && (cost > 0xffffu || instructions > 0xffffu);
    if (j < count) out[j].w = cost | instructions << 16;
  }
  return __any_sync(kFull, bad) ? -1 : count;
}

struct ExactCase {
  int64_t value;
  bool ok;
  uint32_t steps;
};

// Register code on case `c` of every lane (live lanes), by one warp.  `slots`
// is the warp's shared memory, [slot][lane].
//
// The warp runs one instruction at a time for its running lanes.  Lanes whose
// next instruction lies further on -- past a branch the others did not take,
// or out of a loop -- are parked at it (`wait`) and rejoin when the warp
// arrives; the warp always goes to the nearest instruction a lane needs, so
// only control instructions and parked lanes' targets (`join`, the nearest)
// cost anything beyond the operation.  Everything that decides the control
// flow is the same in every lane.
//
// What bounds it: instruction issue and the latency of a dispatch (fetch,
// jump, two shared-memory operands, store).  The stack VM it replaces took
// about 110 machine instructions per dispatch and tested every lane's
// pointer at each; a list search of P = 8192 on 200 cases spent 1650 us per
// round in it and 420 us here.
__device__ __forceinline__ ExactCase run_exact(const VmView& v, const uint4* __restrict__ words, const int64_t* consts,
                                               int c, bool live, int64_t* slots) {
  constexpr int kNone = 0x7fffffff;
  const int lane = threadIdx.x & 31;
  char* const column = reinterpret_cast<char*>(slots + lane);
  auto at = [&](uint32_t slot) -> int64_t& { return *reinterpret_cast<int64_t*>(column + slot * 256u); };
  {
    const uint4 head = __ldg(words);
    for (int j = 0; j < v.n_inputs; ++j)
      if (live) at(j) = __ldg(&v.inputs[size_t(j) * v.C + c]);
    for (uint32_t k = 0; k < (head.x >> 16); ++k) at(head.y + k) = __ldg(&consts[k]);
  }
  const uint4* __restrict__ code = words + 1;
  ExactCase out{0, false, 0};
  int ip = 0, join = kNone, wait = kNone, fuel = v.fuel;
  bool run = live;
  uint4 w = __ldg(code);
  auto charge = [&](bool who) {
    if (who) {
      const int cost = int(w.w & 0xffffu);
      if (fuel < cost) run = false;  // Timeout
      else { fuel -= cost; out.steps += w.w >> 16; }
    }
  };
  charge(run);
  for (;;) {
    const uint4 next = __ldg(code + ip + 1);
    const uint32_t op = w.x & 0xffu;
    const int64_t a = at((w.x >> 8) & 0xffu), b = at((w.x >> 16) & 0xffu);
    int64_t& d = at(w.x >> 24);
    const int target = int(w.y & 0xffffu);
    int dest;
    switch (op) {
#define GB_EXACT(NAME, EXPR) case NAME: if (run) d = (EXPR); goto straight;
      GB_EXACT(X_MOVE, a)
      GB_EXACT(X_IMM, int64_t(uint64_t(w.y) | uint64_t(w.z) << 32))
      GB_EXACT(X_NEG, wrap_neg(a))
      GB_EXACT(X_NOT, a ^ 1)
      GB_EXACT(X_ABS, a < 0 ? wrap_neg(a) : a)
      GB_EXACT(X_LEN, __ldg(&v.lists[a]))
      GB_EXACT(X_ADD, wrap_add(a, b))
      GB_EXACT(X_SUB, wrap_sub(a, b))
      GB_EXACT(X_MUL, wrap_mul(a, b))
      GB_EXACT(X_LT, a < b)
      GB_EXACT(X_LE, a <= b)
      GB_EXACT(X_GT, a > b)
      GB_EXACT(X_GE, a >= b)
      GB_EXACT(X_EQ, a == b)
      GB_EXACT(X_NE, a != b)
      GB_EXACT(X_MIN, a < b ? a : b)
      GB_EXACT(X_MAX, a > b ? a : b)
      GB_EXACT(X_IDIV0, idiv0(a, b))
      GB_EXACT(X_IMOD0, imod0(a, b))
      GB_EXACT(X_TDIV0, tdiv0(a, b))
      GB_EXACT(X_TMOD0, tmod0(a, b))
#undef GB_EXACT
      case X_MOD:
        if (run) {
          if (b == 0) run = false;  // ZeroDiv
          else d = py_mod(a, b);
        }
        goto straight;
      case X_INDEX:
        if (run) {
          const int64_t len = __ldg(&v.lists[a]), j = b < 0 ? b + len : b;  // Python-style negative index
          if (j < 0 || j >= len) run = false;                               // index out of range
          else d = __ldg(&v.lists[a + 1 + j]);
        }
        goto straight;
#define GB_EXACT_SELECT(NAME, CMP)                                            \
  case NAME: {                                                                \
    const bool yes = a CMP b;                                                 \
    const int64_t r = at(yes ? w.y & 0xffu : (w.y >> 8) & 0xffu);             \
    const int extra = int(int16_t(w.z & 0xffffu));                            \
    if (run) {                                                                \
      d = r;                                                                  \
      fuel -= max(yes ? extra : -extra, 0);                                   \
      out.steps += yes ? uint32_t(int(int16_t(w.z >> 16))) : 0u;              \
    }                                                                         \
    goto straight;                                                            \
  }
      GB_EXACT_SELECT(X_SEL_LT, <)
      GB_EXACT_SELECT(X_SEL_LE, <=)
      GB_EXACT_SELECT(X_SEL_GT, >)
      GB_EXACT_SELECT(X_SEL_GE, >=)
      GB_EXACT_SELECT(X_SEL_EQ, ==)
      GB_EXACT_SELECT(X_SEL_NE, !=)
#undef GB_EXACT_SELECT
      case X_BEGIN: case X_BEGIN_REVERSE:
        if (run) {
          const int64_t len = __ldg(&v.lists[a]);
          d = len;
          at((w.x >> 24) - 1) = op == X_BEGIN ? 0 : len - 1;
        }
        goto straight;
      case X_ELEMENT:
        if (run) {
          d = __ldg(&v.lists[at((w.y >> 16) & 0xffu) + 1 + b]);
          at((w.x >> 24) + 1) = wrap_add(at(w.y >> 24), b);
        }
        goto straight;
      default: break;
    }
    {
      // control: `yes` lanes go to the target, the others to the next word
      bool yes = false;
      switch (op) {
        case X_JLT: yes = a < b; break;
        case X_JLE: yes = a <= b; break;
        case X_JGT: yes = a > b; break;
        case X_JGE: yes = a >= b; break;
        case X_JEQ: yes = a == b; break;
        case X_JNE: yes = a != b; break;
        case X_JT: yes = a != 0; break;
        case X_JF: yes = a == 0; break;
        case X_JMP: yes = true; break;
        case X_RET:
          if (run && fuel >= 0) {
            out.value = a;
            out.ok = true;
          }
          run = false;
          break;
        case X_TEST: yes = a <= 0; break;
        case X_NEXT: case X_NEXT_REVERSE: {
          const int64_t cursor = op == X_NEXT ? a + 1 : a - 1;
          yes = op == X_NEXT ? cursor < b : cursor >= 0;
          if (run) {
            at((w.x >> 8) & 0xffu) = cursor;
            if (yes) {
              d = __ldg(&v.lists[at((w.y >> 16) & 0xffu) + 1 + cursor]);
              at((w.x >> 24) + 1) = wrap_add(at(w.y >> 24), cursor);
            }
          }
          break;
        }
        case X_FOR:
          if (run) {
            if (a < 0) run = false;  // a negative bound: a type error
            d = 0;
            if (a > 0) at((w.y >> 16) & 0xffu) = 0;
          }
          yes = a == 0;
          break;
        case X_FOR_NEXT: {
          const int64_t counter = wrap_add(a, 1);
          yes = counter < b;
          if (run) {
            at((w.x >> 8) & 0xffu) = counter;
            if (yes) at((w.y >> 16) & 0xffu) = counter;
          }
          break;
        }
        default: run = false; break;  // X_FAIL: the end of a statement program without a return
      }
      const unsigned going = __ballot_sync(kFull, run && yes), staying = __ballot_sync(kFull, run && !yes);
      const int low = min(target, ip + 1), high = max(target, ip + 1);
      const bool low_is_target = target <= ip;
      const unsigned to_low = low_is_target ? going : staying;
      if (to_low) {
        dest = low;
        if (to_low != (going | staying)) {
          // the lanes bound further on are parked there
          if (run && yes != low_is_target) { run = false; wait = high; }
          join = min(join, high);
        }
      } else if (going | staying) {
        dest = high;
      } else {
        if (join == kNone) break;  // every lane has finished
        dest = join;
      }
      if (dest > join) {
        if (run) { run = false; wait = dest; }
        dest = join;
      }
      w = dest == ip + 1 ? next : __ldg(code + dest);
      ip = dest;
      if (ip == join) {
        if (wait == ip) { run = true; wait = kNone; }
        join = __reduce_min_sync(kFull, wait);
      }
      charge(run);
      continue;
    }
  straight:
    ++ip;
    w = next;
    if (ip == join) {
      const bool back = wait == ip;
      if (back) { run = true; wait = kNone; }
      join = __reduce_min_sync(kFull, wait);
      charge(back);
    }
  }
  return out;
}

}  // namespace gb
