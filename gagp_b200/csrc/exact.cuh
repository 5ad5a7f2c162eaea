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
// instruction, as is a comparison with the branch on it.
//
// A value if that only loads, computes and chooses (no operation of its
// subtree can fail or loop) becomes a select: the cases of a tile disagree on
// most conditions, so the warp would run both branches anyway, and the
// branch, the jump over the other branch and two joins cost more than the
// branches.  What its path costs is decided per case: the select pays for the
// nodes of the branch taken, when every if around it took the branch it is in.
// Those choices are the bits of `paths`, one per nesting level: an if with
// ifs in its branches writes its bit (X_COND) before them and reads it after
// them (X_PICK); one without is a single instruction (X_SELECT).
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

// x: op | a << 8 | b << 16 | d << 24 (slots); y: jump target (its byte offset)
// or select operands (X_SELECT, X_PICK: the path bits of the ifs around it << 16
// and their values on its path << 24; X_COND: its own bit), a traversal's list
// and start slots << 16 and << 24, or the immediate's low half; z: the
// immediate's high half or a select's charges (true, false) and instructions
// (true, false), a byte each; w: charge | instructions << 16 (see above).
enum : uint32_t {
  // dispatched by exact_straight, in the order of its branch targets
  X_MOVE = 0, X_ADD, X_SUB, X_MUL, X_LT, X_LE, X_GT, X_GE, X_EQ, X_NE, X_MIN, X_MAX, X_NEG, X_NOT, X_ABS,
  X_SELECT,                   // + 0..5: on LT .. NE
  X_COND = X_SELECT + 6,      // + 0..5
  X_PICK = X_COND + 6, X_INDEX, X_NEXT, X_FOR_NEXT,
  // straight on, by run_exact
  X_IMM, X_LEN, X_MOD, X_IDIV0, X_IMOD0, X_TDIV0, X_TMOD0, X_BEGIN, X_BEGIN_REVERSE, X_ELEMENT,
  // control, with X_NEXT and X_FOR_NEXT
  X_JUMP,                     // + 0..5: on LT .. NE; + 6: on a true value, + 7: on a false one
  X_NEXT_REVERSE = X_JUMP + 8, X_JMP, X_TEST, X_FOR, X_RET, X_FAIL, X_COUNT
};
static_assert(X_IMM == 31, "exact_straight leaves at operations from 31 on");
__device__ __forceinline__ bool exact_control(uint32_t op) { return op >= X_JUMP || op == X_NEXT || op == X_FOR_NEXT; }

constexpr int kExactSlots = 32;    // slots of a program
constexpr int kExactNarrow = 16;   // slots of most: 4 KB of shared memory per warp (k_vm_exact)
constexpr int kExactConsts = 8;    // of which at most these hold constants
constexpr int kExactWords = 384;   // instructions of a program
constexpr int kExactDepth = 48;    // nesting of a row (below every capacity of the reference's compiler)
// Nodes of an if that is a select: at most 7 nesting levels (an if has at
// least 5 nodes beside its deeper branch), and a byte holds its charges.
constexpr int kSelectNodes = 40;
constexpr int8_t kNoType = GAGP_TAG_INVALID;
constexpr uint32_t kNoSlot = 0xff;  // a traversal whose index is not read (its start), a length not kept in a slot

// Per-warp shared memory of lower_exact_warp.
struct ExactScratch {
  uint32_t fuel[kMaxLowerNodes + 1];   // charges of the nodes before this one
  uint32_t cw[kExactWords];            // a word's charge | instructions << 16 | control << 31
  int16_t end[kMaxLowerNodes];         // one past the subtree
  int16_t words[kMaxLowerNodes + 1];   // words of the nodes before this one
  int16_t start[kMaxLowerNodes];       // open slots; not-flat nodes so far; then the first word's offset from the parent's
  int16_t at[kMaxLowerNodes];          // a traversal's or a let's binder numbers; then the subtree's first word
  uint8_t pos[kMaxLowerNodes];         // temporaries the parent holds while the node runs; then the slot of its value
  uint8_t slot[kMaxLowerNodes];        // temporaries all ancestors hold
  uint32_t ifs[kMaxLowerNodes / 32];   // bit i: node i is an if
  uint8_t par[kMaxLowerNodes], kind[kMaxLowerNodes], flags[kMaxLowerNodes], mark[kMaxLowerNodes];
  // by class: an operation's register operation, an input's or a grammar
  // local's slot, a bound read's binder node, a constant's slot rank (0xff:
  // an immediate), the slot an assignment or a loop stores to
  uint8_t aux[kMaxLowerNodes];
  int8_t type[kMaxLowerNodes];         // completion type (an if's and a let's: type_of)
};

// Node classes.
enum : uint8_t {
  N_CONST = 0, N_SLOT, N_BOUND, N_LEN, N_OP1, N_OP2, N_IF, N_AND, N_OR, N_LET, N_TRAVERSE, N_SEQUENCE, N_NIL, N_ASSIGN, N_RETURN,
  N_FOR, N_BAD
};
// Node flags: the child's number; a comparison its if performs; an if that
// is a select; a node below a select; a comparison; a select with ifs in its
// branches; a bound read: which of the traversal's binders it names (bits 6-7).
enum : uint8_t { NF_ORD = 3, NF_FUSED = 4, NF_SELECT = 8, NF_INSIDE = 16, NF_COMPARE = 32, NF_PICK = 64 };
// Marks: the value goes straight into a slot of the parent; a leaf read where
// it is used (no word, no temporary); a traversal body that is the
// traversal's own state (nothing to do); a traversal whose index is read.
enum : uint8_t { NM_DIRECTED = 1, NM_ALIAS = 2, NM_IDLE = 4, NM_INDEX = 8 };

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
// every lane), or negative when the row takes the reference bytecode instead.
// words: [0] instructions | constants << 16, first constant slot, the list
// inputs whose lengths follow the constants, slots; the instructions follow,
// and one more word may be read past the last.  An IntList input's length
// is read often (a loop bound, every index) and changes only when the program
// assigns the input, so programs that do not keep it in a slot, loaded with
// the inputs, and len of that input is an operand.  `keep` false: no length
// is kept, for a row that fits the slots without them (kTooManySlots: this row
// may be one); 2000 programs of a fold and 11 lengths over 12 list inputs and
// 200 cases took 6.3 ms a call on the interpreter and take 2.0 this way.
//
// What bounds it: latency (a chain of shared-memory passes over the nodes, a
// pass per question; about 40k cycles beside a full round's other warps).
// The bytecode lowering walks the tree on one lane instead: 86 us a range of
// 1024 list-program children against 51 us here.  Every node's words,
// temporaries and charges follow from sums along its path from the root and
// over the nodes before it, as in lower_accumulator_emit, so the lanes share
// the nodes; what several passes ask of a node (its operation, binder, type)
// is kept in shared memory, which took the walk from 143 to 47 us (selects
// cost it 14 us more, taking what words share out of the per-class code gave
// 10 back).
constexpr int kTooManySlots = -2;
__device__ __noinline__ int lower_exact_warp(const SearchDesc& s, const uint64_t* node, int n, const int64_t* cval,
                                             int nc, uint4* words, int word_cap, int64_t* consts, ExactScratch& m,
                                             bool keep, int* slots_out) {
  const int lane = threadIdx.x & 31;
  if (n <= 0 || n > kMaxLowerNodes) return -1;
  const bool statements = is_statement_tag(s.slot_type);
  const int n_inputs = s.local_count;
  if (n_inputs > kExactSlots || s.return_fuel > 0xffu) return -1;
  bool bad = false;
  int named = 0, lets = 0;
  // ---- classes, charges, open slots
  {
    const bool unit = s.unit_fuel;
    uint32_t open = 1, fuel = 0, seen = 0;
#pragma unroll 1
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
        lets += kind == N_LET;
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
  lets = int(__reduce_add_sync(kFull, unsigned(lets)));
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
#pragma unroll 1
  for (int base = 0; base < n; base += 32) {
    const int i = base + lane;
    const int r = i < n ? m.start[i] : 0;
    int e = n;
    bool found = i >= n;
#pragma unroll 1
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
#pragma unroll 1
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
#pragma unroll 1
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
#pragma unroll 1
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
  // ---- what the compiler checks, and which subtrees are flat (loads,
  // operations that cannot fail and ifs over a comparison: a select may run
  // both branches)
  {
    uint32_t not_flat = 0;
#pragma unroll 1
    for (int base = 0; base < n; base += 32) {
      const int i = base + lane;
      bool flat = true;
      if (i < n) {
        const uint8_t kind = m.kind[i];
        const uint32_t op = m.aux[i];
        flat = kind < N_LEN || ((kind == N_OP1 || kind == N_OP2) && op != X_MOD && op != X_INDEX) ||
               (kind == N_IF && (m.flags[i + 1] & NF_COMPARE));
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
            // a bound that is no Int fails at run time too (the bytecode's is_int)
            bad |= type_of(i + 1) != GAGP_TAG_INT || !is_statement_tag(type_of(child(i, 1)));
            break;
          default: break;
        }
        bad |= kind >= N_SEQUENCE && !statements;  // statements only among statements
      }
      const unsigned if_mask = __ballot_sync(kFull, i < n && m.kind[i] == N_IF);
      if (lane == 0) m.ifs[base >> 5] = if_mask;
      uint32_t total;
      const uint32_t before = warp_prefix(i < n && !flat, &total);
      if (i < n) m.start[i] = int16_t(not_flat + before + uint32_t(!flat));  // through node i
      not_flat += total;
    }
    bad |= type_of(0) != s.slot_type && !(statements && is_statement_tag(type_of(0)));
  }
  if (__any_sync(kFull, bad)) return -1;
  // ---- list inputs whose lengths are kept
  uint32_t kept = 0;
  {
    uint32_t assigned = 0, read = 0;
#pragma unroll 1
    for (int i = lane; i < n; i += 32) {
      const uint8_t kind = m.kind[i];
      if ((kind == N_ASSIGN || kind == N_FOR) && m.aux[i] < n_inputs) assigned |= 1u << m.aux[i];
      if (((kind == N_OP1 && m.aux[i] == X_LEN) || (kind == N_OP2 && m.aux[i] == X_INDEX) || kind == N_TRAVERSE) &&
          m.kind[i + 1] == N_SLOT && m.aux[i + 1] < n_inputs)
        read |= 1u << m.aux[i + 1];
    }
    kept = keep ? __reduce_or_sync(kFull, read) & ~__reduce_or_sync(kFull, assigned) : 0u;
  }
  auto kept_length = [&](int i) -> bool { return m.kind[i] == N_SLOT && m.aux[i] < n_inputs && (kept >> m.aux[i] & 1u); };
  __syncwarp();
#pragma unroll 1
  for (int i = lane; i < n; i += 32)
    if (m.kind[i] == N_OP1 && m.aux[i] == X_LEN && kept_length(i + 1)) m.kind[i] = N_LEN;
  // a search's rows are definitely assigned: generation, crossover, mutation
  // and import each keep only such rows; rows to be scored may be any
  if (statements && s.errors) {
    bool ok = false;
    if (lane == 0) ok = row_locals_defined(s, node, n);
    if (!__shfl_sync(kFull, ok, 0)) return -1;
  }
  __syncwarp();
  // the first if in [from, end), else end
  auto next_if = [&](int from, int end) -> int {
    for (int word = from >> 5; word * 32 < end; ++word) {
      uint32_t bits = m.ifs[word];
      if (word == from >> 5) bits &= ~0u << (from & 31);
      if (bits) return min(word * 32 + __ffs(bits) - 1, end);
    }
    return end;
  };
  // ---- fused comparisons and selects
#pragma unroll 1
  for (int i = lane; i < n; i += 32) {
    if (m.kind[i] != N_IF) continue;
    const int c0 = i + 1, c1 = m.end[c0], end = m.end[i];
    if (!(m.flags[c0] & NF_COMPARE)) continue;
    m.flags[c0] |= NF_FUSED;
    if (m.start[end - 1] != m.start[i] || end - i > kSelectNodes || is_statement_tag(type_of(c1))) continue;
    if (!s.unit_fuel) {
      uint32_t charge = m.fuel[end] - m.fuel[i];
      for (int j = i; j < end; j = next_if(j + 1, end)) charge += ex_of(j).merge_fuel;
      if (charge > 0xffu) continue;
    }
    m.flags[i] |= uint8_t(NF_SELECT | (next_if(c1, end) < end ? NF_PICK : 0));
  }
  __syncwarp();
#pragma unroll 1
  for (int i = lane; i < n; i += 32) {
    bool inside = false;
    for (int x = i; x > 0 && !inside; x = m.par[x]) inside = m.kind[m.par[x]] == N_IF && (m.flags[m.par[x]] & NF_SELECT);
    if (inside) m.flags[i] |= NF_INSIDE;
  }
  __syncwarp();
  auto alias = [&](int i) -> bool { return m.mark[i] & NM_ALIAS; };
  // ---- words
  uint32_t total_words = 0;
#pragma unroll 1
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
      const bool leaf_read = !directed && (kind == N_SLOT || kind == N_BOUND || kind == N_LEN || (kind == N_CONST && m.aux[i] != 0xff));
      const bool idle = kind == N_BOUND && above == N_TRAVERSE && ord == 3 && m.aux[i] == p && (flags >> 6) == 2;
      m.mark[i] = uint8_t((directed ? NM_DIRECTED : 0) | (leaf_read ? NM_ALIAS : 0) | (idle ? NM_IDLE : 0));
      switch (kind) {
        case N_CONST: case N_SLOT: case N_BOUND: case N_LEN: own = !leaf_read && !idle; break;
        case N_OP1: case N_OP2: own = !(flags & NF_FUSED); break;
        case N_IF: own = (flags & (NF_SELECT | NF_PICK)) == NF_SELECT ? 1 : 2; break;
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
#pragma unroll 1
  for (int k = lane; k < count; k += 32) m.cw[k] = 0;
  __syncwarp();
#pragma unroll 1
  for (int i = lane; i < n; i += 32)
    if (m.kind[i] == N_BOUND && m.kind[m.aux[i]] == N_TRAVERSE && (m.flags[i] >> 6) == 1) m.mark[m.aux[i]] |= NM_INDEX;
  __syncwarp();
  auto size = [&](int i) { return m.words[m.end[i]] - m.words[i]; };
  // ---- first words and temporaries: offsets from the parent, then sums
  // along the path from the root
#pragma unroll 1
  for (int i = lane; i < n; i += 32) {
    if (i == 0) { m.start[0] = 0; m.pos[0] = 0; }
    const int a = w_arity(node[i]);
    const uint8_t kind = m.kind[i];
    const bool select = kind == N_IF && (m.flags[i] & NF_SELECT), pick = select && (m.flags[i] & NF_PICK);
    int at = 0, held = kind == N_TRAVERSE ? 5 : 0;
    for (int x = 0, c = i + 1; x < a; ++x, c = m.end[c]) {
      if (select && !pick && x == 1) {
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
          at += pick ? x == 0 : !select && x < 2;
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
#pragma unroll 1
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
  // The reference's compiler refuses a row with more open lets or live locals
  // than its tables hold.  A let's value holds none of these slots while it
  // runs, so of lets a row can nest more than that; the open traversals and
  // loops are bounded by the slots (5 T + 2 F + inputs and locals <= 32), and
  // what the compiler holds for them by 32 + 4 T <= 56 of its 64 locals, so
  // up to 8 lets fit without counting.
  static_assert(kExactSlots == 32 && kLowerLocals == 64 && kLowerLets >= 8, "rows of few lets are not counted");
  if (lets > 8) {
#pragma unroll 1
    for (int i = lane; i < n; i += 32) {
      int open = 0, locals = base_slot;
      for (int x = m.par[i], child_of = i; child_of > 0; child_of = x, x = m.par[x]) {
        const uint8_t kind = m.kind[x];
        open += kind == N_LET;
        locals += kind == N_LET ? 1 : kind == N_TRAVERSE ? 9 : kind == N_FOR ? 2 : 0;
      }
      bad |= open > kLowerLets || locals > kLowerLocals;
    }
  }
  const int const_base = base_slot + __reduce_max_sync(kFull, top);
  const int length_base = const_base + const_count, slots = length_base + __popc(kept);
  if (__any_sync(kFull, bad)) return -1;
  if (slots > kExactSlots) return kept ? kTooManySlots : -1;
  __syncwarp();
  // ---- every node writes its words
  uint4* out = words + 1;
  auto fuel_of = [&](int i) -> uint32_t { return m.fuel[i + 1] - m.fuel[i]; };
  auto length_slot = [&](int i) -> uint32_t {  // of list input i (kNoSlot: not kept)
    return kept_length(i) ? uint32_t(length_base + __popc(kept & ((1u << m.aux[i]) - 1))) : kNoSlot;
  };
  auto leaf_slot = [&](int i) -> uint32_t {
    const uint8_t kind = m.kind[i];
    const int aux = m.aux[i];
    if (kind == N_LEN) return length_slot(i + 1);
    if (kind == N_CONST) return uint32_t(const_base + aux);
    if (kind == N_SLOT) return uint32_t(aux);
    const int which = m.flags[i] >> 6;  // of a traversal: 0 element, 1 index, 2 state
    return uint32_t(base_slot + m.slot[aux] + (m.kind[aux] == N_LET || which == 2 ? 0 : 3 + which));
  };
#pragma unroll 1
  for (int i = lane; i < n; i += 32) m.pos[i] = uint8_t(alias(i) ? leaf_slot(i) : uint32_t(base_slot + m.slot[i]));
  __syncwarp();
  auto operand = [&](int i) -> uint32_t { return m.pos[i]; };
  // charge and instructions of a node that is read (a kept length: the input's load and len)
  auto read_cost = [&](int i) -> uint32_t {
    return m.kind[i] == N_LEN ? (m.fuel[i + 2] - m.fuel[i]) | 2u << 16 : fuel_of(i) | 1u << 16;
  };
  auto leaf_cost = [&](int i) -> uint32_t { return alias(i) ? read_cost(i) : 0u; };
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
  // a word's byte offset, as jumps name it
  auto offset = [](int k) -> uint32_t { return uint32_t(k) * uint32_t(sizeof(uint4)); };
  auto put = [&](int k, uint32_t op, uint32_t a, uint32_t b, uint32_t d, uint32_t y, uint32_t z, uint32_t cost) {
    out[k] = make_uint4(op | a << 8 | b << 16 | d << 24, y, z, 0);
    atomicAdd(&m.cw[k], cost + (exact_control(op) ? 1u << 31 : 0u));
  };
  int rank = 0;
#pragma unroll 1
  for (int base = 0; base < n; base += 32) {
    const int i = base + lane;
    const bool live = i < n;
    const uint8_t kind = live ? m.kind[i] : uint8_t(N_NIL);
    const unsigned const_mask = __ballot_sync(kFull, kind == N_CONST);
    const int row_const = rank + __popc(const_mask & ((1u << lane) - 1));
    rank += __popc(const_mask);
    if (!live) continue;
    // what most words need of a node, by all lanes together: its children,
    // its first two operands (an if over a comparison: the comparison's) with
    // the charges of their reads, and where the value goes
    const int at = m.at[i], words_of = size(i);
    const uint8_t flags = m.flags[i], aux = m.aux[i];
    const bool inside = flags & NF_INSIDE;
    const int arity = w_arity(node[i]);
    const int c0 = arity > 0 ? i + 1 : i, c1 = arity > 1 ? int(m.end[c0]) : i, c2 = arity > 2 ? int(m.end[c1]) : i;
    const bool fused = kind == N_IF && (m.flags[c0] & NF_FUSED);
    const int l = fused ? c0 + 1 : c0, r = fused ? int(m.end[l]) : kind == N_IF ? i : c1;
    const uint32_t a = operand(l), b = arity > 1 ? operand(r) : 0u, to = target_slot(i), store = store_cost(i);
    uint32_t own = inside ? 0u : read_cost(i);
    if (!inside && (arity == 1 || arity == 2) && kind >= N_OP1) own += leaf_cost(c0) + (arity == 2 ? leaf_cost(c1) : 0u);
    switch (kind) {
      case N_CONST:
        if (alias(i)) break;
        if (aux != 0xff) {
          put(at, X_MOVE, leaf_slot(i), 0, to, 0, 0, own + store);
        } else {
          const uint64_t v = uint64_t(cval[row_const]);
          put(at, X_IMM, 0, 0, to, uint32_t(v), uint32_t(v >> 32), own + store);
        }
        break;
      case N_SLOT: case N_BOUND: case N_LEN:
        if (!(m.mark[i] & (NM_ALIAS | NM_IDLE))) put(at, X_MOVE, leaf_slot(i), 0, to, 0, 0, own + store);
        break;
      case N_OP1: case N_OP2:
        if (flags & NF_FUSED) break;
        put(at + words_of - 1, aux, a, arity == 2 ? b : 0u, to, aux == X_INDEX ? length_slot(c0) : 0u, 0, own + store);
        break;
      case N_IF: {
        const uint32_t merge_fuel = s.unit_fuel ? 1u : ex_of(i).merge_fuel;
        uint32_t cost = (fuel_of(i) | 1u << 16) + leaf_cost(l) + store, compare = X_COUNT;
        if (fused) {
          cost += (fuel_of(c0) | 1u << 16) + leaf_cost(r);
          compare = m.aux[c0] - X_LT;
        }
        if (flags & NF_SELECT) {
          // what this if pays when its path is taken: itself, its comparison
          // and the nodes of the branch taken, except what ifs below it pay
          uint32_t pay[2];
#pragma unroll
          for (int branch = 0; branch < 2; ++branch) {
            uint32_t charge = fuel_of(i) + fuel_of(c0), instructions = 2;
            if (branch == 0) {
              charge += merge_fuel;
              ++instructions;
            }
            const int from = branch == 0 ? c1 : c2, end = m.end[from];
            charge += m.fuel[c1] - m.fuel[c0 + 1] + m.fuel[end] - m.fuel[from];
            instructions += uint32_t(c1 - c0 - 1 + end - from);
            for (int part = 0; part < 2; ++part) {
              const int last = part ? end : c1;
              for (int j = next_if(part ? from : c0 + 1, last); j < last; j = next_if(m.end[j], last)) {
                charge -= m.fuel[m.end[j]] - m.fuel[j];
                instructions -= uint32_t(m.end[j] - j);
              }
            }
            pay[branch] = charge | instructions << 16;
          }
          // the ifs around it, nearest first into the highest bit
          uint32_t values = 0, bits = 0;
          for (int x = i; x > 0; x = m.par[x]) {
            const int p = m.par[x], ord = m.flags[x] & NF_ORD;
            if (m.kind[p] == N_IF && !(m.flags[p] & NF_SELECT)) break;
            if (m.kind[p] == N_IF && ord > 0) {
              values = values << 1 | uint32_t(ord == 1);
              bits = bits << 1 | 1u;
            } else if (m.kind[p] != N_IF && m.kind[p] != N_OP1 && m.kind[p] != N_OP2) {
              break;
            }
          }
          const uint32_t y = operand(c1) | operand(c2) << 8 | bits << 16 | values << 24;
          const uint32_t z = (pay[0] & 0xffu) | (pay[1] & 0xffu) << 8 | (pay[0] >> 16) << 16 | (pay[1] >> 16) << 24;
          if (flags & NF_PICK) {
            put(at + size(c0), X_COND + compare, a, b, 0, bits + 1, 0, 0);
            put(at + words_of - 1, X_PICK, 0, 0, to, y, z, store);
          } else {
            put(at + words_of - 1, X_SELECT + compare, a, b, to, y, z, store);
          }
          break;
        }
        // jump over the first branch when the condition does not hold:
        // LT/LE/GT/GE and EQ/NE inverted
        const uint32_t jump = compare == X_COUNT ? 7u : compare < 4 ? 3u - compare : 9u - compare;
        put(at + size(c0), X_JUMP + jump, a, fused ? b : 0u, 0, offset(m.at[c2]), 0, cost);
        put(m.at[c2] - 1, X_JMP, 0, 0, 0, offset(at + words_of), 0, merge_fuel | 1u << 16);
        break;
      }
      case N_AND: case N_OR: {
        const int last = at + words_of - 1;
        put(at + size(c0), X_JUMP + (kind == N_AND ? 7u : 6u), a, 0, 0, offset(last), 0,
            read_cost(i) + leaf_cost(c0) + store);
        put(last - 1, X_JMP, 0, 0, 0, offset(last + 1), 0, 3 * fuel_of(i) + (3u << 16));
        put(last, X_IMM, 0, 0, to, kind == N_OR, 0, fuel_of(i) | 1u << 16);
        break;
      }
      case N_TRAVERSE: {
        const RegionInfo& info = s.regions[ex_of(i).operand];
        const bool reverse = info.traversal == 2;
        // an event's charge and instructions (lower_code's walk_after)
        auto event = [&](int which, uint32_t instructions) -> uint32_t {
          return (info.fuel_profile ? info.event_cost[which] : instructions) + (instructions << 16);
        };
        const uint32_t q = uint32_t(base_slot + m.slot[i]);  // state, cursor, limit, element, index
        const int c3 = m.end[c2];
        const uint32_t views = a << 16 | (m.mark[i] & NM_INDEX ? b : kNoSlot) << 24;
        const int next = m.at[c3] + size(c3);
        // the result's read happens once, when the traversal completes: paid here
        put(at + size(c0) + size(c1), reverse ? X_BEGIN_REVERSE : X_BEGIN, a, 0, q + 2, length_slot(c0), 0,
            leaf_cost(c0) + leaf_cost(c1) + event(4, 1) + event(5, 1) + event(8, 3) + event(11, 3) + event(14, 2) +
                event(15, 2) + event(25, 1) + store);
        put(m.at[c3] - 2, X_TEST, q + 2, 0, 0, offset(next + 1), 0, event(16, 1) + event(17, reverse ? 4 : 2) + event(18, 4));
        put(m.at[c3] - 1, X_ELEMENT, 0, q + 1, q + 3, views, 0, 0);
        // paid on entry to the body, by the first pass and by every next one
        atomicAdd(&m.cw[m.at[c3]], event(19, 3) + event(20, 1) + event(21, 4));
        put(next, reverse ? X_NEXT_REVERSE : X_NEXT, q + 1, q + 2, q + 3, offset(m.at[c3]) | views, 0,
            event(22, 1) + event(23, 4) + event(24, 1) + event(18, 4) + (m.mark[c3] & NM_IDLE ? fuel_of(c3) | 1u << 16 : 0u));
        if (m.mark[i] & NM_DIRECTED) put(next + 1, X_MOVE, q, 0, to, 0, 0, 0);
        break;
      }
      case N_RETURN:
        put(at + words_of - 1, X_RET, a, 0, 0, 0, 0, own);
        break;
      case N_FOR: {
        // lower_code's template, every instruction charged 1
        const uint32_t q = uint32_t(base_slot + m.slot[i]);  // bound, counter
        const int next = m.at[c1] + size(c1);
        const uint32_t user = uint32_t(aux) << 16;
        put(m.at[c1] - 1, X_FOR, q, 0, q + 1, offset(next + 1) | user, 0, 14 + (14u << 16));
        atomicAdd(&m.cw[m.at[c1]], 2 + (2u << 16));
        put(next, X_FOR_NEXT, q + 1, q, 0, offset(m.at[c1]) | user, 0, 9 + (9u << 16));
        break;
      }
      default: break;
    }
  }
  if (lane == 0) {
    if (statements) put(count - 1, X_FAIL, 0, 0, 0, 0, 0, 0);
    else put(count - 1, X_RET, operand(0), 0, 0, 0, 0, (s.return_fuel | 1u << 16) + leaf_cost(0));
    words[0] = make_uint4(uint32_t(count) | uint32_t(const_count) << 16, uint32_t(const_base), kept, uint32_t(slots));
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
  *slots_out = slots;
  return __any_sync(kFull, bad) ? -1 : count;
}

struct ExactCase {
  int64_t value;
  bool ok;
  uint32_t steps;
};

// Shared memory by its 32-bit address.
__device__ __forceinline__ int64_t lds64(uint32_t at) {
  int64_t v;
  asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(at));
  return v;
}
__device__ __forceinline__ void sts64(uint32_t at, int64_t v) { asm volatile("st.shared.b64 [%0], %1;" ::"r"(at), "l"(v)); }

// Runs instructions from the word (x, y) at `pc` for the lanes with `run` set,
// up to the first one that run_exact executes (X_IMM on; an index into a list
// whose length is not kept; a loop's last step) or to the word whose address's
// low half is `join` (odd: none); pc and (x, y) are then that word.  Lanes that
// leave a loop before the others are parked at the next word: `wait` is its
// offset and it becomes the join, since no join lies before it.  All lanes
// run the same instructions.
//
// PTX, because every branch here is uniform and the compiler cannot know: a
// switch in C++ becomes a tree of comparisons with a convergence barrier at
// each branch, 76 instructions per dispatch in all (17 of them branches) on
// the initial programs of a list search.  Here an operation is one indirect
// branch to its handler and one back.
//
// Operands: %0 x, %1 y, %2 pc, %3 run, %4 fuel, %5 steps, %6 paths, %7 the
// lane's column of slots, %8 lists, %9 code, %10 wait, %11 join.  Slot k lies 256 k bytes
// into the column: one byte permutation moves a slot field to bits 8..15.
__device__ __forceinline__ void exact_straight(uint2& w, uint64_t& pc, uint32_t& run, int& fuel, uint32_t& steps,
                                               uint32_t& paths, uint32_t column, const int64_t* lists, uint64_t code,
                                               int& wait, uint32_t& join) {
  asm volatile(
      "{\n"
      "  .reg .pred r, p, q, k;\n"
      "  .reg .b32 op, fa, fb, fd, nx, ny, t, z, u, m;\n"
      "  .reg .b64 a, b, v, g;\n"
      "  T: .branchtargets V0, V1, V2, V3, V4, V5, V6, V7, V8, V9, V10, V11, V12, V13, V14, S0, S1, S2, S3, S4, S5,\n"
      "     C0, C1, C2, C3, C4, C5, P0, I0, X0, W0, OUT;\n"
      "  setp.ne.u32 r, %3, 0;\n"
      "L:\n"
      "  and.b32 op, %0, 255;\n"
      "  ld.v2.b32 {nx, ny}, [%2+16];\n"
      "  prmt.b32 fa, %0, 0, 0x4414;\n"
      "  prmt.b32 fb, %0, 0, 0x4424;\n"
      "  prmt.b32 fd, %0, 0, 0x4434;\n"
      "  add.u32 fa, fa, %7;\n"
      "  add.u32 fb, fb, %7;\n"
      "  add.u32 fd, fd, %7;\n"
      "  ld.shared.b64 a, [fa];\n"
      "  ld.shared.b64 b, [fb];\n"
      "  min.u32 op, op, 31;\n"
      "  brx.idx.uni op, T;\n"
      "V0: @r st.shared.b64 [fd], a; bra.uni N;\n"
      "V1: add.s64 v, a, b; @r st.shared.b64 [fd], v; bra.uni N;\n"
      "V2: sub.s64 v, a, b; @r st.shared.b64 [fd], v; bra.uni N;\n"
      "V3: mul.lo.s64 v, a, b; @r st.shared.b64 [fd], v; bra.uni N;\n"
      "V4: setp.lt.s64 p, a, b; selp.b64 v, 1, 0, p; @r st.shared.b64 [fd], v; bra.uni N;\n"
      "V5: setp.le.s64 p, a, b; selp.b64 v, 1, 0, p; @r st.shared.b64 [fd], v; bra.uni N;\n"
      "V6: setp.gt.s64 p, a, b; selp.b64 v, 1, 0, p; @r st.shared.b64 [fd], v; bra.uni N;\n"
      "V7: setp.ge.s64 p, a, b; selp.b64 v, 1, 0, p; @r st.shared.b64 [fd], v; bra.uni N;\n"
      "V8: setp.eq.s64 p, a, b; selp.b64 v, 1, 0, p; @r st.shared.b64 [fd], v; bra.uni N;\n"
      "V9: setp.ne.s64 p, a, b; selp.b64 v, 1, 0, p; @r st.shared.b64 [fd], v; bra.uni N;\n"
      "V10: min.s64 v, a, b; @r st.shared.b64 [fd], v; bra.uni N;\n"
      "V11: max.s64 v, a, b; @r st.shared.b64 [fd], v; bra.uni N;\n"
      "V12: neg.s64 v, a; @r st.shared.b64 [fd], v; bra.uni N;\n"
      "V13: xor.b64 v, a, 1; @r st.shared.b64 [fd], v; bra.uni N;\n"
      "V14: abs.s64 v, a; @r st.shared.b64 [fd], v; bra.uni N;\n"
      "S0: setp.lt.s64 p, a, b; bra.uni SEL;\n"
      "S1: setp.le.s64 p, a, b; bra.uni SEL;\n"
      "S2: setp.gt.s64 p, a, b; bra.uni SEL;\n"
      "S3: setp.ge.s64 p, a, b; bra.uni SEL;\n"
      "S4: setp.eq.s64 p, a, b; bra.uni SEL;\n"
      "S5: setp.ne.s64 p, a, b; bra.uni SEL;\n"
      "C0: setp.lt.s64 p, a, b; bra.uni CND;\n"
      "C1: setp.le.s64 p, a, b; bra.uni CND;\n"
      "C2: setp.gt.s64 p, a, b; bra.uni CND;\n"
      "C3: setp.ge.s64 p, a, b; bra.uni CND;\n"
      "C4: setp.eq.s64 p, a, b; bra.uni CND;\n"
      "C5: setp.ne.s64 p, a, b;\n"
      "CND:\n"  // paths with bit y set to the condition
      "  or.b32 t, %6, %1;\n"
      "  not.b32 u, %1;\n"
      "  and.b32 u, %6, u;\n"
      "  selp.b32 %6, t, u, p;\n"
      "  bra.uni N;\n"
      "P0:\n"  // the path bit above the bits of the ifs around
      "  bfe.u32 m, %1, 16, 8;\n"
      "  add.u32 m, m, 1;\n"
      "  and.b32 m, m, %6;\n"
      "  setp.ne.u32 p, m, 0;\n"
      "SEL:\n"
      "  ld.b32 z, [%2+8];\n"
      "  prmt.b32 t, %1, 0, 0x4404;\n"
      "  prmt.b32 u, %1, 0, 0x4414;\n"
      "  selp.b32 t, t, u, p;\n"
      "  add.u32 t, t, %7;\n"
      "  ld.shared.b64 v, [t];\n"
      "  shr.u32 m, %1, 24;\n"
      "  xor.b32 m, m, %6;\n"
      "  shr.u32 u, %1, 16;\n"
      "  and.b32 m, m, u;\n"
      "  and.b32 m, m, 255;\n"
      "  setp.eq.and.u32 k, m, 0, r;\n"
      "  selp.b32 t, 0x4440, 0x4441, p;\n"
      "  selp.b32 u, 0x4442, 0x4443, p;\n"
      "  prmt.b32 t, z, 0, t;\n"
      "  prmt.b32 u, z, 0, u;\n"
      "  @k sub.s32 %4, %4, t;\n"
      "  @k add.u32 %5, %5, u;\n"
      "  @r st.shared.b64 [fd], v;\n"
      "  bra.uni N;\n"
      "I0:\n"  // a's element b, a negative b from the end; out of range fails
      "  setp.eq.u32 p, %1, 255;\n"
      "  @p bra.uni OUT;\n"
      "  shl.b32 t, %1, 8;\n"
      "  add.u32 t, t, %7;\n"
      "  ld.shared.b64 v, [t];\n"
      "  add.s64 g, b, v;\n"
      "  setp.lt.s64 p, b, 0;\n"
      "  selp.b64 b, g, b, p;\n"
      "  setp.lt.and.u64 r, b, v, r;\n"
      "  add.s64 a, a, b;\n"
      "  shl.b64 a, a, 3;\n"
      "  add.s64 a, a, %8;\n"
      "  @r ld.global.nc.b64 v, [a+8];\n"
      "  @r st.shared.b64 [fd], v;\n"
      "  bra.uni N;\n"
      "X0:\n"  // a traversal's step
      "  add.s64 v, a, 1;\n"
      "  setp.lt.and.s64 p, v, b, r;\n"
      "  vote.sync.any.pred q, p, 0xffffffff;\n"
      "  @!q bra.uni OUT;\n"
      "  not.pred k, p;\n"
      "  and.pred k, k, r;\n"
      "  prmt.b32 t, %1, 0, 0x4424;\n"
      "  add.u32 t, t, %7;\n"
      "  ld.shared.b64 g, [t];\n"
      "  add.s64 g, g, v;\n"
      "  shl.b64 g, g, 3;\n"
      "  add.s64 g, g, %8;\n"
      "  @p ld.global.nc.b64 a, [g+8];\n"
      "  @p st.shared.b64 [fa], v;\n"
      "  shr.u32 u, %1, 24;\n"
      "  setp.eq.u32 q, u, 255;\n"
      "  @q bra.uni X1;\n"
      "  prmt.b32 t, %1, 0, 0x4434;\n"
      "  add.u32 t, t, %7;\n"
      "  ld.shared.b64 b, [t];\n"
      "  add.s64 b, b, v;\n"
      "  @p st.shared.b64 [fd+256], b;\n"
      "X1:\n"
      "  @p st.shared.b64 [fd], a;\n"
      "  bra.uni BACK;\n"
      "W0:\n"  // a for_range's step: counter a, bound b, the variable's slot in y
      "  add.s64 v, a, 1;\n"
      "  setp.lt.and.s64 p, v, b, r;\n"
      "  vote.sync.any.pred q, p, 0xffffffff;\n"
      "  @!q bra.uni OUT;\n"
      "  not.pred k, p;\n"
      "  and.pred k, k, r;\n"
      "  prmt.b32 t, %1, 0, 0x4424;\n"
      "  add.u32 t, t, %7;\n"
      "  @p st.shared.b64 [fa], v;\n"
      "  @p st.shared.b64 [t], v;\n"
      "BACK:\n"  // lanes k leave the loop, lanes p go on at the target
      "  vote.sync.any.pred q, k, 0xffffffff;\n"
      "  @!q bra.uni B1;\n"
      "  cvt.u32.u64 t, %2;\n"
      "  add.u32 %11, t, 16;\n"
      "  cvt.u32.u64 u, %9;\n"
      "  sub.u32 u, %11, u;\n"
      "  @k mov.b32 %10, u;\n"
      "  and.pred r, r, p;\n"
      "B1:\n"
      "  and.b32 t, %1, 65535;\n"
      "  cvt.u64.u32 g, t;\n"
      "  add.s64 %2, %9, g;\n"
      "  ld.b32 z, [%2+12];\n"
      "  ld.v2.b32 {%0, %1}, [%2];\n"
      "  and.b32 t, z, 65535;\n"
      "  sub.s32 t, %4, t;\n"
      "  setp.ge.and.s32 r, t, 0, r;\n"
      "  shr.u32 u, z, 16;\n"
      "  @r mov.b32 %4, t;\n"
      "  @r add.u32 %5, %5, u;\n"
      "  bra.uni L;\n"
      "N:\n"
      "  add.s64 %2, %2, 16;\n"
      "  mov.b32 %0, nx;\n"
      "  mov.b32 %1, ny;\n"
      "  cvt.u32.u64 t, %2;\n"
      "  setp.ne.u32 p, t, %11;\n"
      "  @p bra.uni L;\n"
      "OUT:\n"
      "  selp.u32 %3, 1, 0, r;\n"
      "}"
      : "+r"(w.x), "+r"(w.y), "+l"(pc), "+r"(run), "+r"(fuel), "+r"(steps), "+r"(paths),
        "+r"(column), "+l"(lists), "+l"(code), "+r"(wait), "+r"(join)
      :
      : "memory");
}

// Register code on case `c` of every lane (live lanes), by one warp.  `slots`
// is the warp's shared memory, [slot][lane]; `code` the instructions, in
// shared memory or in place.
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
// round in it, 365 us in this VM with its straight code in C++ and ifs as
// branches, and 235 us now, 78% of the issue slots taken.
__device__ __forceinline__ ExactCase run_exact(const VmView& v, const uint4* code, uint4 head, const int64_t* consts,
                                               int c, bool live, const int64_t* slots) {
  constexpr int kNone = 0x7fffffff, kWord = int(sizeof(uint4));
  const uint32_t column = uint32_t(__cvta_generic_to_shared(slots + (threadIdx.x & 31)));
  const uint64_t base = reinterpret_cast<uint64_t>(code);
  auto get = [&](uint32_t slot256) { return lds64(column + slot256); };
  auto set = [&](uint32_t slot256, int64_t value) { sts64(column + slot256, value); };
  auto field_a = [](uint32_t x) { return __byte_perm(x, 0, 0x4414); };
  auto field_b = [](uint32_t x) { return __byte_perm(x, 0, 0x4424); };
  auto field_d = [](uint32_t x) { return __byte_perm(x, 0, 0x4434); };
  auto word = [&](int offset) { return *reinterpret_cast<const uint2*>(reinterpret_cast<const char*>(code) + offset); };
  for (int j = 0; j < v.n_inputs; ++j)
    if (live) set(256u * j, __ldg(&v.inputs[size_t(j) * v.C + c]));
  for (uint32_t k = 0; k < (head.x >> 16); ++k) set(256u * (head.y + k), __ldg(&consts[k]));
  for (uint32_t kept = head.z, k = head.y + (head.x >> 16); kept; kept &= kept - 1, ++k)
    if (live) set(256u * k, __ldg(&v.lists[get(256u * (__ffs(kept) - 1))]));
  ExactCase out{0, false, 0};
  int ip = 0, join = kNone, wait = kNone, fuel = v.fuel;  // ip, join, wait: byte offsets
  uint32_t paths = 0;  // the branches of the selects around this instruction
  bool run = live;
  // lanes `who` arrive at word `ip`: they pay through its next control word
  auto charge = [&](bool who) {
    const uint32_t paid = reinterpret_cast<const uint32_t*>(reinterpret_cast<const char*>(code) + ip)[3];
    if (who) {
      const int left = fuel - int(paid & 0xffffu);
      if (left < 0) {
        run = false;  // Timeout
      } else {
        fuel = left;
        out.steps += paid >> 16;
      }
    }
  };
  uint2 w = word(0);
  charge(run);
  for (;;) {
    {
      uint64_t pc = base + uint64_t(ip);
      uint32_t running = run, join_at = join == kNone ? 1u : uint32_t(base) + uint32_t(join);
      __syncwarp();
      exact_straight(w, pc, running, fuel, out.steps, paths, column, v.lists, base, wait, join_at);
      run = running != 0;
      ip = int(uint32_t(pc) - uint32_t(base));
      join = join_at & 1u ? kNone : int(join_at - uint32_t(base));
    }
    bool pays = false;
    if (ip != join) {
      const uint32_t op = w.x & 0xffu;
      const int64_t a = get(field_a(w.x)), b = get(field_b(w.x));
      const int target = int(w.y & 0xffffu);
      int dest = ip + kWord;
      if (!exact_control(op)) {
        // straight on
        if (run) {
          const uint32_t d = field_d(w.x);
          if (op == X_ELEMENT) {
            set(d, __ldg(&v.lists[get(field_b(w.y)) + 1 + b]));
            if (w.y >> 24 != kNoSlot) set(d + 256u, wrap_add(get(field_d(w.y)), b));
          } else if (op == X_BEGIN || op == X_BEGIN_REVERSE) {
            const int64_t len = w.y == kNoSlot ? __ldg(&v.lists[a]) : get(w.y * 256u);
            set(d, len);
            set(d - 256u, op == X_BEGIN ? 0 : len - 1);
          } else if (op == X_IMM) {
            const uint32_t high = reinterpret_cast<const uint32_t*>(reinterpret_cast<const char*>(code) + ip)[2];
            set(d, int64_t(uint64_t(w.y) | uint64_t(high) << 32));
          } else if (op == X_LEN) {
            set(d, __ldg(&v.lists[a]));
          } else if (op == X_INDEX) {
            const int64_t len = __ldg(&v.lists[a]), j = b < 0 ? b + len : b;  // Python-style negative index
            if (j < 0 || j >= len) run = false;                               // index out of range
            else set(d, __ldg(&v.lists[a + 1 + j]));
          } else if (op == X_MOD) {
            if (b == 0) run = false;  // ZeroDiv
            else set(d, py_mod(a, b));
          } else if (op <= X_IMOD0) {
            set(d, op == X_IDIV0 ? idiv0(a, b) : imod0(a, b));
          } else {
            set(d, op == X_TDIV0 ? tdiv0(a, b) : tmod0(a, b));
          }
        }
      } else {
        if (op <= X_FOR_NEXT || op == X_NEXT_REVERSE) {
          // a loop's step: lanes that go on jump back.  A parked lane waits
          // past the loop or further on in its body, so the jump meets none.
          bool go;
          if (op == X_FOR_NEXT) {
            const int64_t counter = wrap_add(a, 1);
            go = run && counter < b;
            if (go) {
              set(field_a(w.x), counter);
              set(field_b(w.y), counter);
            }
          } else {
            const bool reverse = op == X_NEXT_REVERSE;
            const int64_t cursor = reverse ? a - 1 : a + 1;
            go = run && (reverse ? cursor >= 0 : cursor < b);
            if (go) {
              set(field_d(w.x), __ldg(&v.lists[get(field_b(w.y)) + 1 + cursor]));
              if (w.y >> 24 != kNoSlot) set(field_d(w.x) + 256u, wrap_add(get(field_d(w.y)), cursor));
              set(field_a(w.x), cursor);
            }
          }
          const bool stay = run && !go;
          if (__any_sync(kFull, go)) {
            if (__any_sync(kFull, stay)) {
              if (stay) {
                run = false;
                wait = dest;
              }
              join = min(join, dest);
            }
            dest = target;
          } else if (!__any_sync(kFull, stay)) {
            dest = kNone;
          }
        } else if (op >= X_RET) {
          if (op == X_RET && run && fuel >= 0) {
            out.value = a;
            out.ok = true;
          }
          run = false;  // X_FAIL: the end of a statement program without a return
          dest = kNone;
        } else {
          // a forward branch
          bool yes = true;
          if (op < X_JUMP + 6) {
            const uint32_t relation = a < b ? 1u : a == b ? 2u : 4u;  // LT 1, LE 3, GT 4, GE 6, EQ 2, NE 5
            yes = relation & (0x526431u >> (4 * (op - X_JUMP)));
          } else if (op < X_NEXT_REVERSE) {
            yes = (a != 0) == (op == X_JUMP + 6);
          } else if (op != X_JMP) {
            yes = a <= 0;  // X_TEST: an empty list
            if (op == X_FOR && run) {
              if (a < 0) run = false;  // a negative bound: a type error
              set(field_d(w.x), 0);
              if (a > 0) set(field_b(w.y), 0);
            }
          }
          const bool go = run && yes, stay = run && !yes;
          if (__any_sync(kFull, stay)) {
            if (__any_sync(kFull, go)) {
              if (go) {
                run = false;
                wait = target;
              }
              join = min(join, target);
            }
          } else {
            dest = __any_sync(kFull, go) ? target : kNone;
            if (dest > join && run) {
              run = false;
              wait = dest;
            }
          }
        }
        dest = min(dest, join);
        if (dest == kNone) break;  // every lane has finished
        pays = run;
      }
      ip = dest;
      w = word(ip);
    }
    if (ip == join) {
      if (wait == ip) {
        run = pays = true;
        wait = kNone;
      }
      join = __reduce_min_sync(kFull, wait);
    }
    if (__any_sync(kFull, pays)) charge(pays);
  }
  return out;
}

}  // namespace gb
