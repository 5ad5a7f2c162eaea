// The accumulator VM: one warp runs one straight-line accumulator program
// (lower.cuh) on tiles of 32 K cases; lane l holds cases tile + 32 k + l for
// k < K (coalesced input loads).  The program's staged code, its constants
// and the temporaries live in the warp's shared memory; with one or two
// inputs (NIN) the tile's input values live in registers, otherwise (NIN 0)
// they are read through L1.  The semantics are vm.cuh's.
#pragma once
#include "vm.cuh"

namespace gb {

// Staged form of an accumulator instruction: one handler per (operation,
// operand class), chosen once when a warp stages a program, so that running
// an instruction costs one jump.  Swapped operands are normalised away (a
// swapped comparison is the mirrored one; subtraction has a reversed
// handler).  Word x: handler | for SELECT the three 2-bit operand kinds << 8,
// for OUT what leaves the loop (OutCode << 8, the operand's kind << 16).
// Word y: the operand's shared address (temporaries: without the lane's
// part), an input's index, or SELECT's three 8-bit indices.
enum : uint32_t {
  H_MOV = 0,  // + class: temporary, constant, input (of two: the first), second input
  H_SPILL = 4, H_NEG, H_NOT, H_ABS, H_SELECT, H_OUT,
  H_BINARY = 10  // + 4 * binary operation + class
};
enum : uint32_t {
  HB_ADD = 0, HB_SUB, HB_RSUB, HB_MUL, HB_LT, HB_LE, HB_GT, HB_GE, HB_EQ, HB_NE, HB_AND, HB_OR, HB_MIN, HB_MAX,
  HB_COUNT
};
// What leaves the dispatch loop: the divisions, whose code the compiler
// expands, and the program's end.
enum OutCode : uint32_t {
  OUT_IDIV0 = 0, OUT_RIDIV0, OUT_IMOD0, OUT_RIMOD0, OUT_TDIV0, OUT_RTDIV0, OUT_TMOD0, OUT_RTMOD0, OUT_END
};

// How an operation (| swap << 5) is staged: its first handler, or the out
// code | 64; bit 7 set when the handler goes by the operand's class.
constexpr int kStageEntries = 64;
constexpr uint32_t kStageOut = 64, kStageClass = 128;
__device__ inline uint32_t stage_entry(int index) {
  const bool swap = index & 32;
  auto binary = [](uint32_t b) { return kStageClass | (H_BINARY + 4 * b); };
  switch (index & 31) {
    case A_MOV: return kStageClass | H_MOV;
    case A_SPILL: return H_SPILL;
    case A_NEG: return H_NEG;
    case A_NOT: return H_NOT;
    case A_ABS: return H_ABS;
    case A_SELECT: return H_SELECT;
    case A_ADD: return binary(HB_ADD);
    case A_SUB: return binary(swap ? HB_RSUB : HB_SUB);
    case A_MUL: return binary(HB_MUL);
    case A_LT: return binary(swap ? HB_GT : HB_LT);
    case A_LE: return binary(swap ? HB_GE : HB_LE);
    case A_GT: return binary(swap ? HB_LT : HB_GT);
    case A_GE: return binary(swap ? HB_LE : HB_GE);
    case A_EQ: return binary(HB_EQ);
    case A_NE: return binary(HB_NE);
    case A_AND: return binary(HB_AND);
    case A_OR: return binary(HB_OR);
    case A_MIN: return binary(HB_MIN);
    case A_MAX: return binary(HB_MAX);
    case A_IDIV0: return kStageOut | (swap ? OUT_RIDIV0 : OUT_IDIV0);
    case A_IMOD0: return kStageOut | (swap ? OUT_RIMOD0 : OUT_IMOD0);
    case A_TDIV0: return kStageOut | (swap ? OUT_RTDIV0 : OUT_TDIV0);
    case A_TMOD0: return kStageOut | (swap ? OUT_RTMOD0 : OUT_TMOD0);
    default: return kStageOut | OUT_END;  // no such operation
  }
}
static_assert(H_BINARY + 4 * HB_COUNT <= 128 && OUT_END < 64, "stage entries are seven bits and the class flag");
// Bytes of one temporary (K cases of 32 lanes); a lane's own part of it: two
// cases side by side, so that one 16-byte access moves two.
template <int K>
constexpr uint32_t kTempBytes = K * 256;
template <int K>
constexpr uint32_t kTempLane = K == 1 ? 8 : 16;

template <int K, int NIN>
__device__ __forceinline__ uint2 stage_accumulator(uint2 w, const uint8_t* entries, uint32_t temps, uint32_t consts) {
  const uint32_t entry = entries[(w.x & 31u) | ((w.x >> 8 & 1u) << 5)];
  const uint32_t k1 = (w.x >> 9) & 3u, i1 = w.y & 0xffffu;
  if (entry & kStageClass) {
    const uint32_t h = entry & 127u;
    if (k1 == K_CONST) return make_uint2(h + 1, consts + 8 * i1);
    if (k1 == K_INPUT) return make_uint2(h + (NIN == 2 && i1 ? 3 : 2), i1);
    return make_uint2(h, temps + kTempBytes<K> * i1);  // binary and MOV operands are never the accumulator
  }
  if (entry & kStageOut) return make_uint2(H_OUT | ((entry & 63u) << 8) | (k1 << 16), i1);
  if (entry == H_SELECT)
    return make_uint2(H_SELECT | (((w.x >> 9) & 0x3fu) << 8), (i1 & 255u) | ((w.y >> 16 & 255u) << 8) | (w.x & 0xff0000u));
  return make_uint2(entry, temps + kTempBytes<K> * i1);
}

// The dispatch loop over the operations that need no loop or call of their
// own, until an OUT word.  Written in PTX because the compiler turns a switch
// of this size into a tree of compares and branches with a convergence
// barrier around each: 76 instructions per dispatch of four cases a lane,
// against the 4 to 16 of the operation itself.  Here an operation is one
// indirect branch to its handler and one back, and the next word is fetched
// meanwhile.  The warp runs one program: every branch is uniform.
// Bound by instruction issue and the latency of a dispatch: 16384 programs of
// a scalar search on 2000 cases took 257 M warp instructions and 631 us with
// the switch, 178 M and 340 us with this loop, the narrow division below and
// a third resident block (0.39 -> 0.57 instructions per cycle).
//
// Named registers: a<k> the accumulator, i<k> and j<k> the inputs, b<k> and
// e<k> operands, c a constant; t1 the temporaries' base with the lane's part,
// ln that part, kb the constants.
#define GB_EACH1(M, P) M("0", P "0")
#define GB_EACH2(M, P) GB_EACH1(M, P) M("1", P "1")
#define GB_EACH4(M, P) GB_EACH2(M, P) M("2", P "2") M("3", P "3")
#define GB_SAME1(M, P) M("0", P)
#define GB_SAME2(M, P) GB_SAME1(M, P) M("1", P)
#define GB_SAME4(M, P) GB_SAME2(M, P) M("2", P) M("3", P)
#define GB_LOADT1(R, A) "ld.shared.b64 " R "0, [" A "];\n"
#define GB_LOADT2(R, A) "ld.shared.v2.b64 {" R "0, " R "1}, [" A "];\n"
#define GB_LOADT4(R, A) GB_LOADT2(R, A) "ld.shared.v2.b64 {" R "2, " R "3}, [" A "+512];\n"
#define GB_STORET1(R, A) "st.shared.b64 [" A "], " R "0;\n"
#define GB_STORET2(R, A) "st.shared.v2.b64 [" A "], {" R "0, " R "1};\n"
#define GB_STORET4(R, A) GB_STORET2(R, A) "st.shared.v2.b64 [" A "+512], {" R "2, " R "3};\n"
#define GB_OP_MOV(k, B) "mov.b64 a" k ", " B ";\n"
#define GB_OP_ADD(k, B) "add.s64 a" k ", a" k ", " B ";\n"
#define GB_OP_SUB(k, B) "sub.s64 a" k ", a" k ", " B ";\n"
#define GB_OP_RSUB(k, B) "sub.s64 a" k ", " B ", a" k ";\n"
#define GB_OP_MUL(k, B) "mul.lo.s64 a" k ", a" k ", " B ";\n"
#define GB_OP_SET(C, k, B) "setp." C ".s64 p, a" k ", " B ";\n selp.b64 a" k ", 1, 0, p;\n"
#define GB_OP_LT(k, B) GB_OP_SET("lt", k, B)
#define GB_OP_LE(k, B) GB_OP_SET("le", k, B)
#define GB_OP_GT(k, B) GB_OP_SET("gt", k, B)
#define GB_OP_GE(k, B) GB_OP_SET("ge", k, B)
#define GB_OP_EQ(k, B) GB_OP_SET("eq", k, B)
#define GB_OP_NE(k, B) GB_OP_SET("ne", k, B)
#define GB_OP_AND(k, B) "and.b64 a" k ", a" k ", " B ";\n"
#define GB_OP_OR(k, B) "or.b64 a" k ", a" k ", " B ";\n"
#define GB_OP_MIN(k, B) "min.s64 a" k ", a" k ", " B ";\n"
#define GB_OP_MAX(k, B) "max.s64 a" k ", a" k ", " B ";\n"
#define GB_OP_NEG(k, B) "neg.s64 a" k ", a" k ";\n"
#define GB_OP_NOT(k, B) "xor.b64 a" k ", a" k ", 1;\n"
#define GB_OP_ABS(k, B) "abs.s64 a" k ", a" k ";\n"
#define GB_OP_TRUE(k, B) "setp.ne.s64 q" k ", b" k ", 0;\n"
#define GB_OP_PICK(k, B) "selp.b64 a" k ", b" k ", e" k ", q" k ";\n"
#define GB_GOTO_N "bra.uni N;\n"
// One binary operation's handlers: temporary, constant, input, second input.
#define GB_BINARY(K, N, M)                                                     \
  N "0:\n add.u32 t, y, ln;\n" GB_LOADT##K("b", "t") GB_EACH##K(M, "b") GB_GOTO_N \
  N "1:\n ld.shared.b64 c, [y];\n" GB_SAME##K(M, "c") GB_GOTO_N                \
  N "2:\n" GB_INPUT(K, M) GB_GOTO_N                                            \
  N "3:\n" GB_INPUT2(K, M) GB_GOTO_N
// Input operands: held in registers, or (three inputs and more) loaded; a
// lane past the last case reads 0.
#define GB_INPUT_HELD(K, M) GB_EACH##K(M, "i")
#define GB_INPUT2_HELD(K, M) GB_EACH##K(M, "j")
#define GB_FETCH(k, B) "mov.b64 " B ", 0;\n @l" k " ld.global.nc.b64 " B ", [g+256*" k "];\n"
#define GB_INPUT_READ(K, M) "cvt.u64.u32 g, y;\n mad.lo.u64 g, g, cs, ib;\n" GB_EACH##K(GB_FETCH, "b") GB_EACH##K(M, "b")
#define GB_NONE(K, M)
// SELECT's operands: kind z (accumulator, temporary, input, constant), index t.
#define GB_MOVE_B(k, B) "mov.b64 b" k ", " B ";\n"
#define GB_MOVE_E(k, B) "mov.b64 e" k ", " B ";\n"
#define GB_OPERAND(K, N, R, MOVE)                                              \
  N "T: .branchtargets " N "A, " N "M, " N "I, " N "C;\n"                      \
  "brx.idx.uni z, " N "T;\n"                                                   \
  N "A:\n" GB_EACH##K(MOVE, "a") "bra.uni " N "N;\n"                           \
  N "M:\n mad.lo.u32 t, t, tb, t1;\n" GB_LOADT##K(R, "t") "bra.uni " N "N;\n"  \
  N "I:\n" GB_SELECT_INPUT(K, R, MOVE) "bra.uni " N "N;\n"                     \
  N "C:\n mad.lo.u32 t, t, 8, kb;\n ld.shared.b64 c, [t];\n" GB_SAME##K(MOVE, "c") \
  N "N:\n"
#define GB_SELECT_INPUT_ONE(K, R, MOVE) GB_EACH##K(MOVE, "i")
#define GB_EITHER_B(k, B) "selp.b64 b" k ", i" k ", j" k ", p;\n"
#define GB_EITHER_E(k, B) "selp.b64 e" k ", i" k ", j" k ", p;\n"
#define GB_SELECT_INPUT_TWO(K, R, MOVE) "setp.eq.u32 p, t, 0;\n" GB_EITHER_##MOVE(K)
#define GB_EITHER_GB_MOVE_B(K) GB_EACH##K(GB_EITHER_B, "b")
#define GB_EITHER_GB_MOVE_E(K) GB_EACH##K(GB_EITHER_E, "e")
#define GB_SELECT_INPUT_READ(K, R, MOVE) "cvt.u64.u32 g, t;\n mad.lo.u64 g, g, cs, ib;\n" GB_EACH##K(GB_FETCH, R)
#define GB_DISPATCH_REGS                                                                                  \
  "  .reg .pred p, q0, q1, q2, q3;\n"                                                                    \
  "  .reg .b32 op, x, y, nx, ny, t, z, pc;\n"                                                            \
  "  .reg .b64 b0, b1, b2, b3, e0, e1, e2, e3, c, g;\n"
#define GB_DISPATCH(K, TABLE3)                                                                           \
  "  T: .branchtargets MOV0, MOV1, MOV2, " TABLE3("MOV") "SPILL, NEG, NOT, ABS, SELECT, OUT,\n"          \
  "     ADD0, ADD1, ADD2, " TABLE3("ADD") "SUB0, SUB1, SUB2, " TABLE3("SUB") "RSB0, RSB1, RSB2, "        \
  TABLE3("RSB") "MUL0, MUL1, MUL2, " TABLE3("MUL") "LT0, LT1, LT2, " TABLE3("LT") "LE0, LE1, LE2, "      \
  TABLE3("LE") "GT0, GT1, GT2, " TABLE3("GT") "GE0, GE1, GE2, " TABLE3("GE") "EQ0, EQ1, EQ2, "           \
  TABLE3("EQ") "NE0, NE1, NE2, " TABLE3("NE") "AND0, AND1, AND2, " TABLE3("AND") "OR0, OR1, OR2, "       \
  TABLE3("OR") "MIN0, MIN1, MIN2, " TABLE3("MIN") "MAX0, MAX1, MAX2, " TABLE3("MAX") "OUT;\n"            \
  "  mov.b32 pc, %2;\n"                                                                                  \
  "  ld.shared.v2.b32 {x, y}, [pc];\n"                                                                   \
  "L:\n"                                                                                                 \
  "  ld.shared.v2.b32 {nx, ny}, [pc+8];\n"                                                               \
  "  add.u32 pc, pc, 8;\n"                                                                               \
  "  and.b32 op, x, 255;\n"                                                                              \
  "  brx.idx.uni op, T;\n"                                                                               \
  GB_BINARY(K, "MOV", GB_OP_MOV)                                                                         \
  "SPILL:\n add.u32 t, y, ln;\n" GB_STORET##K("a", "t") GB_GOTO_N                                        \
  "NEG:\n" GB_EACH##K(GB_OP_NEG, "a") GB_GOTO_N                                                          \
  "NOT:\n" GB_EACH##K(GB_OP_NOT, "a") GB_GOTO_N                                                          \
  "ABS:\n" GB_EACH##K(GB_OP_ABS, "a") GB_GOTO_N                                                          \
  GB_BINARY(K, "ADD", GB_OP_ADD) GB_BINARY(K, "SUB", GB_OP_SUB) GB_BINARY(K, "RSB", GB_OP_RSUB)          \
  GB_BINARY(K, "MUL", GB_OP_MUL) GB_BINARY(K, "LT", GB_OP_LT) GB_BINARY(K, "LE", GB_OP_LE)               \
  GB_BINARY(K, "GT", GB_OP_GT) GB_BINARY(K, "GE", GB_OP_GE) GB_BINARY(K, "EQ", GB_OP_EQ)                 \
  GB_BINARY(K, "NE", GB_OP_NE) GB_BINARY(K, "AND", GB_OP_AND) GB_BINARY(K, "OR", GB_OP_OR)               \
  GB_BINARY(K, "MIN", GB_OP_MIN) GB_BINARY(K, "MAX", GB_OP_MAX)                                          \
  "SELECT:\n bfe.u32 z, x, 8, 2;\n and.b32 t, y, 255;\n" GB_OPERAND(K, "SC", "b", GB_MOVE_B)             \
  GB_EACH##K(GB_OP_TRUE, "b")                                                                            \
  "  bfe.u32 z, x, 10, 2;\n bfe.u32 t, y, 8, 8;\n" GB_OPERAND(K, "ST", "b", GB_MOVE_B)                   \
  "  bfe.u32 z, x, 12, 2;\n bfe.u32 t, y, 16, 8;\n" GB_OPERAND(K, "SE", "e", GB_MOVE_E)                  \
  GB_EACH##K(GB_OP_PICK, "a")                                                                            \
  "N:\n"                                                                                                 \
  "  mov.b32 x, nx;\n"                                                                                   \
  "  mov.b32 y, ny;\n"                                                                                   \
  "  bra.uni L;\n"                                                                                       \
  "OUT:\n"                                                                                               \
  "  mov.b32 %0, x;\n mov.b32 %1, y;\n mov.b32 %2, pc;\n"

// Operands: %0 x, %1 y, %2 pc, %3 t1, %4 ln, %5 kb, %6 bytes of a temporary,
// then the accumulators and the inputs (or where they are read: the first
// input's address at the lane's first case, the bytes from one input to the
// next, the live cases' bits).
#define GB_ENTER1 ".reg .b64 a0;\n mov.b64 a0, %7;\n mov.b32 t1, %3; mov.b32 ln, %4; mov.b32 kb, %5; mov.b32 tb, %6;\n"
#define GB_LEAVE1 "mov.b64 %7, a0;\n"
#define GB_ENTER_I1 ".reg .b64 i0;\n mov.b64 i0, %8;\n"
#define GB_ENTER_J1 ".reg .b64 j0;\n mov.b64 j0, %9;\n"
#define GB_ENTER_R1 ".reg .pred l0;\n .reg .b64 ib, cs;\n mov.b64 ib, %8; mov.b64 cs, %9;\n and.b32 t, %10, 1; setp.ne.u32 l0, t, 0;\n"
#define GB_ACC1 "+l"(acc[0])
#define GB_REG1(V) "l"(V[0])
#define GB_ENTER2 ".reg .b64 a0, a1;\n mov.b64 a0, %7; mov.b64 a1, %8;\n mov.b32 t1, %3; mov.b32 ln, %4; mov.b32 kb, %5; mov.b32 tb, %6;\n"
#define GB_LEAVE2 "mov.b64 %7, a0; mov.b64 %8, a1;\n"
#define GB_ENTER_I2 ".reg .b64 i0, i1;\n mov.b64 i0, %9; mov.b64 i1, %10;\n"
#define GB_ENTER_J2 ".reg .b64 j0, j1;\n mov.b64 j0, %11; mov.b64 j1, %12;\n"
#define GB_ENTER_R2 ".reg .pred l0, l1;\n .reg .b64 ib, cs;\n mov.b64 ib, %9; mov.b64 cs, %10;\n and.b32 t, %11, 1; setp.ne.u32 l0, t, 0; and.b32 t, %11, 2; setp.ne.u32 l1, t, 0;\n"
#define GB_ACC2 "+l"(acc[0]), "+l"(acc[1])
#define GB_REG2(V) "l"(V[0]), "l"(V[1])
#define GB_ENTER4 ".reg .b64 a0, a1, a2, a3;\n mov.b64 a0, %7; mov.b64 a1, %8; mov.b64 a2, %9; mov.b64 a3, %10;\n mov.b32 t1, %3; mov.b32 ln, %4; mov.b32 kb, %5; mov.b32 tb, %6;\n"
#define GB_LEAVE4 "mov.b64 %7, a0; mov.b64 %8, a1; mov.b64 %9, a2; mov.b64 %10, a3;\n"
#define GB_ENTER_I4 ".reg .b64 i0, i1, i2, i3;\n mov.b64 i0, %11; mov.b64 i1, %12; mov.b64 i2, %13; mov.b64 i3, %14;\n"
#define GB_ENTER_J4 ".reg .b64 j0, j1, j2, j3;\n mov.b64 j0, %15; mov.b64 j1, %16; mov.b64 j2, %17; mov.b64 j3, %18;\n"
#define GB_ENTER_R4 ".reg .pred l0, l1, l2, l3;\n .reg .b64 ib, cs;\n mov.b64 ib, %11; mov.b64 cs, %12;\n and.b32 t, %13, 1; setp.ne.u32 l0, t, 0; and.b32 t, %13, 2; setp.ne.u32 l1, t, 0; and.b32 t, %13, 4; setp.ne.u32 l2, t, 0; and.b32 t, %13, 8; setp.ne.u32 l3, t, 0;\n"
#define GB_ACC4 "+l"(acc[0]), "+l"(acc[1]), "+l"(acc[2]), "+l"(acc[3])
#define GB_REG4(V) "l"(V[0]), "l"(V[1]), "l"(V[2]), "l"(V[3])

struct AccumulatorAt {
  uint32_t x, y, pc;          // the word that left the loop, and the next one's shared address
  uint32_t temps, lane_part;  // the temporaries' address with the lane's part, and that part
  uint32_t consts;
};
#define GB_RUN(K, ENTER_INPUTS, TABLE3, INPUTS)                                                           \
  asm volatile("{\n .reg .b32 t1, ln, kb, tb;\n" GB_ENTER##K GB_DISPATCH_REGS ENTER_INPUTS               \
               GB_DISPATCH(K, TABLE3) GB_LEAVE##K "}"                                                     \
               : "+r"(w.x), "+r"(w.y), "+r"(w.pc), "+r"(w.temps), "+r"(w.lane_part), "+r"(w.consts),      \
                 "+r"(temp_bytes), GB_ACC##K                                                              \
               : INPUTS                                                                                   \
               : "memory")
#define GB_TABLE3_NONE(N) "OUT, "
#define GB_TABLE3_TWO(N) N "3, "
#define GB_COMMA ,

#define GB_INPUT GB_INPUT_HELD
#define GB_INPUT2 GB_NONE
#define GB_SELECT_INPUT GB_SELECT_INPUT_ONE
template <int K>
__device__ __forceinline__ void dispatch_one(AccumulatorAt& w, int64_t* acc, const int64_t* in0) {
  uint32_t temp_bytes = kTempBytes<K>;
  if constexpr (K == 1) GB_RUN(1, GB_ENTER_I1, GB_TABLE3_NONE, GB_REG1(in0));
  else if constexpr (K == 2) GB_RUN(2, GB_ENTER_I2, GB_TABLE3_NONE, GB_REG2(in0));
  else GB_RUN(4, GB_ENTER_I4, GB_TABLE3_NONE, GB_REG4(in0));
}
#undef GB_INPUT
#undef GB_INPUT2
#undef GB_SELECT_INPUT

#define GB_INPUT GB_INPUT_HELD
#define GB_INPUT2 GB_INPUT2_HELD
#define GB_SELECT_INPUT GB_SELECT_INPUT_TWO
template <int K>
__device__ __forceinline__ void dispatch_two(AccumulatorAt& w, int64_t* acc, const int64_t* in0, const int64_t* in1) {
  uint32_t temp_bytes = kTempBytes<K>;
  if constexpr (K == 1) GB_RUN(1, GB_ENTER_I1 GB_ENTER_J1, GB_TABLE3_TWO, GB_REG1(in0) GB_COMMA GB_REG1(in1));
  else if constexpr (K == 2) GB_RUN(2, GB_ENTER_I2 GB_ENTER_J2, GB_TABLE3_TWO, GB_REG2(in0) GB_COMMA GB_REG2(in1));
  else GB_RUN(4, GB_ENTER_I4 GB_ENTER_J4, GB_TABLE3_TWO, GB_REG4(in0) GB_COMMA GB_REG4(in1));
}
#undef GB_INPUT
#undef GB_INPUT2
#undef GB_SELECT_INPUT

#define GB_INPUT GB_INPUT_READ
#define GB_INPUT2 GB_NONE
#define GB_SELECT_INPUT GB_SELECT_INPUT_READ
template <int K>
__device__ __forceinline__ void dispatch_read(AccumulatorAt& w, int64_t* acc, const int64_t* inputs, uint64_t stride,
                                              uint32_t live) {
  uint32_t temp_bytes = kTempBytes<K>;
  if constexpr (K == 1) GB_RUN(1, GB_ENTER_R1, GB_TABLE3_NONE, "l"(inputs) GB_COMMA "l"(stride) GB_COMMA "r"(live));
  else if constexpr (K == 2) GB_RUN(2, GB_ENTER_R2, GB_TABLE3_NONE, "l"(inputs) GB_COMMA "l"(stride) GB_COMMA "r"(live));
  else GB_RUN(4, GB_ENTER_R4, GB_TABLE3_NONE, "l"(inputs) GB_COMMA "l"(stride) GB_COMMA "r"(live));
}
#undef GB_INPUT
#undef GB_INPUT2
#undef GB_SELECT_INPUT

// Division of operands in [-2^30, 2^30) without branches: most of a program's
// values are small, and the compiler's 32- and 64-bit divisions behind a test
// per lane run both where the lanes of a warp differ.  From the float
// reciprocal's estimate and two remainders: a float, its reciprocal and their
// product are each within 2^-22 of their value, so the first quotient is
// within 1/2 + |a / b| 2^-20 and leaves a remainder of at most |b| / 2 + 2^10;
// the second quotient is then within 1/2 + 2^-9 of what is left, and the last
// remainder r = a - q b smaller than |b|.  Its sign is not settled: the
// functions below move it to the one they want.  With b = 0 the results mean
// nothing.
__host__ __device__ __forceinline__ uint32_t outside_narrow(int64_t v) {  // nonzero outside the range
  const uint64_t u = uint64_t(v) + (1ULL << 30);
  return uint32_t(u >> 32) | (uint32_t(u) & 0x80000000u);
}
__device__ __forceinline__ void narrow_divide(int a, int b, int& q, int& r) {
  float inverse;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inverse) : "f"(float(b)));
  const int q1 = __float2int_rn(float(a) * inverse);
  const int left = int(uint32_t(a) - uint32_t(q1) * uint32_t(b));
  const int q2 = __float2int_rn(float(left) * inverse);
  r = int(uint32_t(left) - uint32_t(q2) * uint32_t(b));
  q = int(uint32_t(q1) + uint32_t(q2));
}
// The remainder of the divisor's sign (Python's modulo).
__device__ __forceinline__ int narrow_mod(int r, int b) { return r != 0 && (r ^ b) < 0 ? r + b : r; }
// The remainder of the dividend's sign and the truncated quotient: one
// divisor further where r has the other sign.
__device__ __forceinline__ int narrow_rem(int r, int a, int b) {
  return r != 0 && (r ^ a) < 0 ? ((a ^ b) < 0 ? r - b : r + b) : r;
}
__device__ __forceinline__ int narrow_quot(int q, int r, int a, int b) {
  return r != 0 && (r ^ a) < 0 ? ((a ^ b) < 0 ? q + 1 : q - 1) : q;
}

// A program in the warp's shared memory, ready to run on tiles.
struct VmWarpSmem {
  int64_t* temps;
  uint2* code;
  int64_t* consts;
};

// Stages slot `slot`'s program; `entries` holds stage_entry(0 .. 63).
template <int K, int NIN>
__device__ __forceinline__ void stage_program(const SearchDesc& s, int slot, const VmWarpSmem& w,
                                              const uint8_t* entries, int len) {
  const int lane = threadIdx.x & 31;
  const uint2* code = s.code + size_t(slot) * s.code_stride;
  const int64_t* kpool = s.kpool + size_t(slot) * s.stride;
  const uint32_t temps = uint32_t(__cvta_generic_to_shared(w.temps));
  const uint32_t consts = uint32_t(__cvta_generic_to_shared(w.consts));
  __syncwarp();  // the program before is done with these words
  for (int i = lane; i < len; i += 32) w.code[i] = stage_accumulator<K, NIN>(code[i], entries, temps, consts);
  if (lane < 2) w.code[len + lane] = make_uint2(H_OUT | (OUT_END << 8), 0);  // the end, and the word fetched past it
  for (int i = lane; i < s.stride; i += 32) w.consts[i] = kpool[i];
  __syncwarp();
}

// Runs the staged program on cases [case_begin, case_end), at most 32 K.
template <int K, int NIN>
__device__ __forceinline__ void run_accumulator(const SearchDesc& s, const VmWarpSmem& sm, uint32_t case_begin, uint32_t case_end,
                                                int64_t& loss, uint32_t& wrong) {
  const int lane = threadIdx.x & 31;
  const int C = s.C;  // input-major stride
  const int64_t* __restrict__ inputs = s.inputs;
  int64_t in0[K], in1[K], want[K], acc[K];
  uint32_t live = 0;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const uint32_t c = case_begin + k * 32 + lane;
    const bool on = c < case_end;
    live |= uint32_t(on) << k;
    in0[k] = (NIN >= 1 && on) ? __ldg(&inputs[c]) : 0;
    in1[k] = (NIN >= 2 && on) ? __ldg(&inputs[size_t(C) + c]) : 0;
    want[k] = on ? __ldg(&s.expected[c]) : 0;
    acc[k] = 0;
  }
  AccumulatorAt w;
  w.lane_part = kTempLane<K> * lane;
  w.temps = uint32_t(__cvta_generic_to_shared(sm.temps)) + w.lane_part;
  w.consts = uint32_t(__cvta_generic_to_shared(sm.consts));
  w.pc = uint32_t(__cvta_generic_to_shared(sm.code));
  for (;;) {
    if constexpr (NIN == 1) dispatch_one<K>(w, acc, in0);
    else if constexpr (NIN == 2) dispatch_two<K>(w, acc, in0, in1);
    else dispatch_read<K>(w, acc, inputs + case_begin + lane, uint64_t(C) * 8, live);
    const uint32_t out = (w.x >> 8) & 63u;
    if (out >= OUT_END) break;
    int64_t b[K];
    const uint32_t kind = (w.x >> 16) & 3u;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      if (kind == K_TEMP) {
        b[k] = K == 1 ? sm.temps[w.y * 32 + lane] : sm.temps[w.y * (K * 32) + (k >> 1) * 64 + 2 * lane + (k & 1)];
      } else if (kind == K_CONST) {
        b[k] = sm.consts[w.y];
      } else if (NIN != 0) {
        b[k] = NIN == 2 && w.y ? in1[k] : in0[k];
      } else {
        b[k] = live >> k & 1 ? __ldg(&inputs[size_t(w.y) * C + (case_begin + k * 32 + lane)]) : 0;
      }
    }
    if (out & 1u) {  // reversed operands
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const int64_t a = acc[k];
        acc[k] = b[k];
        b[k] = a;
      }
    }
    uint32_t wide = 0;
#pragma unroll
    for (int k = 0; k < K; ++k) wide |= outside_narrow(acc[k]) | outside_narrow(b[k]);
    if (__any_sync(0xffffffffu, wide != 0)) {
#define GB_ACC_OUT(CODE, OP)                                     \
  case CODE:                                                     \
    _Pragma("unroll") for (int k = 0; k < K; ++k) acc[k] = OP(acc[k], b[k]); \
    break;
      switch (out & ~1u) {
        GB_ACC_OUT(OUT_IDIV0, idiv0)
        GB_ACC_OUT(OUT_IMOD0, imod0)
        GB_ACC_OUT(OUT_TDIV0, tdiv0)
        GB_ACC_OUT(OUT_TMOD0, tmod0)
        default: break;
      }
#undef GB_ACC_OUT
    } else {
      int q[K], r[K];
#pragma unroll
      for (int k = 0; k < K; ++k) narrow_divide(int(acc[k]), int(b[k]), q[k], r[k]);
      if ((out & ~1u) == OUT_IMOD0) {
#pragma unroll
        for (int k = 0; k < K; ++k) acc[k] = int(b[k]) == 0 ? 0 : narrow_mod(r[k], int(b[k]));
      } else if ((out & ~1u) == OUT_TMOD0) {
#pragma unroll
        for (int k = 0; k < K; ++k) acc[k] = int(b[k]) == 0 ? 0 : narrow_rem(r[k], int(acc[k]), int(b[k]));
      } else {
#pragma unroll
        for (int k = 0; k < K; ++k) acc[k] = int(b[k]) == 0 ? 0 : narrow_quot(q[k], r[k], int(acc[k]), int(b[k]));
      }
    }
    __syncwarp();  // the dispatch loop's branches are the warp's
  }
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (live >> k & 1) loss += case_loss(s, s.result_type, acc[k], want[k], wrong);
}

}  // namespace gb
