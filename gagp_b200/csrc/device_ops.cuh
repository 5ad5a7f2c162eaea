// Device building blocks of the resident search: the grammar RNG, the
// self-describing node word, typed subtree generation and warp-cooperative
// row primitives.  Each function names the reference function whose results
// it reproduces exactly (paths relative to the reference root).
//
// Node word (64 bits), B200-first layout of one phase-tree node:
//   [0,16)  construction expression (the reference's origin)
//   [16,32) 1 + the reference expression that opened the node's grammar
//           site (0: no site) -- the whole PhaseGeneSite is a function of it
//   [32,40) depth (root = 1), [40,48) site depth: grammar sites on the path
//           from the root down to and including this node
//   [48,52) arity, [52] constant, [53,64) crossover class of the site
//           (nonterminal and scope; kNoClass: none or variation disabled)
// Storing depth and site depth turns the reference's sequential stack walks
// (phase_node_depth, phase_site_depth, phase_tree_depth) into lookups and
// warp max-reductions: a splice shifts the donor subtree's depths by the
// difference at the splice point and leaves every other node's unchanged.
#pragma once
#include <cstdint>

#include "search_state.h"

namespace gb {

// PhaseExpressionKind / PhaseTreeKind / status codes (reference enums).
enum { EK_OPERATION = 0, EK_CONSTANT = 1, EK_BOUND = 2, EK_REFERENCE = 3, EK_INPUT = 4, EK_ALIAS = 5 };
enum { TK_CONSTANT = 0, TK_LOCAL = 1, TK_OPERATION = 2, TK_IF = 3, TK_AND = 4, TK_OR = 5, TK_PROGRAM = 6,
       TK_BLOCK = 7, TK_NIL = 8, TK_ASSIGN = 9, TK_RETURN = 10, TK_FOR_RANGE = 11, TK_VAR = 12, TK_LET = 13,
       TK_BOUND = 14, TK_REGION = 15, TK_TRAVERSE = 16 };
// Completion tag of a statement (kPhaseStatement,
// cpp/src/evolution/repro/gpu/device/phase_compile.cuh:23): a node or phase
// type, never a runtime value.  Tables narrowed to int8_t keep it as -16.
constexpr int kStatementTag = 0xF0;
__host__ __device__ __forceinline__ bool is_statement_tag(int t) { return (t & 0xff) == kStatementTag; }
constexpr int kNamedLocals = 16;  // grammar locals a phase can name (kPhaseNamedLocals)
enum { ST_OK = 0, ST_INVALID = 1, ST_UNSUPPORTED = 2, ST_CAPACITY = 3 };
constexpr int kFixedSite = 1 << 30;
constexpr uint32_t kNoClass = 0x7ffu;
constexpr unsigned kFull = 0xffffffffu;

// ---------------------------------------------------------------- RNG
// Ranges up to kSmallBound (site counts, value lists, small integer
// domains) draw with 32-bit arithmetic only (Rng::bounded).
constexpr uint64_t kSmallBound = uint64_t(1) << 16;

// A range u of 1 .. 2^16 and what a bounded draw over it needs.  With
// m = 2^32 mod u, a draw v = hi * 2^32 + lo has v mod u =
// ((hi mod u) * m + lo mod u) mod u, and the rejection bound (2^64 - u) mod u is
// m^2 mod u (every intermediate below 2^32).  One division gives
// q = floor((2^32 - 1) / u); floor(x q / 2^32) is then at most one below
// floor(x / u), because q >= 2^32 / u - 1.
struct SmallRange {
  uint32_t u, q, m;
  __device__ __forceinline__ explicit SmallRange(uint32_t range) : u(range), q(0xffffffffu / range) {
    const uint32_t t = 0xffffffffu - q * u;
    m = t + 1 == u ? 0 : t + 1;
  }
  __device__ __forceinline__ uint32_t mod(uint32_t x) const {
    const uint32_t r = x - __umulhi(x, q) * u;
    return r >= u ? r - u : r;
  }
};

__device__ __forceinline__ uint64_t splitmix_next(uint64_t& state) {
  uint64_t v = (state += 0x9e3779b97f4a7c15ULL);
  v = (v ^ (v >> 30)) * 0xbf58476d1ce4e5b9ULL;
  v = (v ^ (v >> 27)) * 0x94d049bb133111ebULL;
  return v ^ (v >> 31);
}
// A draw below `upper` past 2^16, out of line: two 64-bit divisions.
struct Drawn {
  uint64_t value, state;
};
__device__ __noinline__ Drawn draw_wide(uint64_t state, uint64_t upper) {
  const uint64_t threshold = (0 - upper) % upper;
  for (;;) {
    const uint64_t v = splitmix_next(state);
    if (v >= threshold) return Drawn{v % upper, state};
  }
}

// SplitMix64 stream with rejection-sampled bounds
// (DGrammarRandom, cpp/src/evolution/repro/gpu/device/grammar_random.cuh:10-51).
struct Rng {
  uint64_t state;
  __device__ explicit Rng(uint64_t seed) : state(seed) {}
  __device__ __forceinline__ uint64_t next() { return splitmix_next(state); }
  // 32-bit arithmetic only, with no table load on the dependent chain; only a
  // draw below 2^16 can be below the rejection bound
  __device__ __forceinline__ uint32_t bounded(const SmallRange& r) {
    for (;;) {
      const uint64_t v = next();
      if (v < kSmallBound && v < r.mod(r.m * r.m)) continue;
      return r.mod(r.mod(uint32_t(v >> 32)) * r.m + r.mod(uint32_t(v)));
    }
  }
  __device__ __forceinline__ uint64_t bounded(uint64_t upper) {
    if (upper - 1 < uint64_t(kSmallBound)) return bounded(SmallRange(uint32_t(upper)));
    const Drawn d = draw_wide(state, upper);
    state = d.state;
    return d.value;
  }
  // bounded(upper) for a fixed upper with its rejection bound
  // ((2^64 - upper) mod upper) and magic floor((2^64 - 1) / upper) given:
  // the residue comes from a multiply-high quotient estimate, at most two
  // below the true quotient, and at most two corrections
  __device__ __forceinline__ uint64_t bounded_fixed(uint64_t upper, uint64_t threshold, uint64_t magic) {
    for (;;) {
      const uint64_t v = next();
      if (v >= threshold) {
        uint64_t r = v - __umul64hi(v, magic) * upper;
        while (r >= upper) r -= upper;
        return r;
      }
    }
  }
  // 53-bit uniform in [0,1): exact (a power-of-two scale)
  __device__ __forceinline__ double unit() { return __dmul_rn(double(next() >> 11), 0x1.0p-53); }
};

__device__ __forceinline__ uint64_t mix64(uint64_t x) {
  x += 0x9e3779b97f4a7c15ULL;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ULL;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebULL;
  return x ^ (x >> 31);
}

// ---------------------------------------------------------------- node words
__host__ __device__ __forceinline__ int w_origin(uint64_t w) { return int(w & 0xffffu); }
__host__ __device__ __forceinline__ int w_entry(uint64_t w) { return int((w >> 16) & 0xffffu) - 1; }
__host__ __device__ __forceinline__ int w_depth(uint64_t w) { return int((w >> 32) & 0xffu); }
__host__ __device__ __forceinline__ int w_sval(uint64_t w) { return int((w >> 40) & 0xffu); }
__host__ __device__ __forceinline__ int w_arity(uint64_t w) { return int((w >> 48) & 0xfu); }
__host__ __device__ __forceinline__ bool w_const(uint64_t w) { return (w >> 52) & 1u; }
__host__ __device__ __forceinline__ uint32_t w_class(uint64_t w) { return uint32_t(w >> 53); }
__host__ __device__ __forceinline__ bool w_site(uint64_t w) { return ((w >> 16) & 0xffffu) != 0; }
__host__ __device__ __forceinline__ uint64_t w_make(int origin, int entry, int depth, int sval, int arity, bool constant,
                                           uint32_t cls) {
  return uint64_t(uint32_t(origin) & 0xffffu) | (uint64_t(uint32_t(entry + 1) & 0xffffu) << 16) |
         (uint64_t(uint32_t(depth) & 0xffu) << 32) | (uint64_t(uint32_t(sval) & 0xffu) << 40) |
         (uint64_t(uint32_t(arity) & 0xfu) << 48) | (uint64_t(constant) << 52) | (uint64_t(cls & 0x7ffu) << 53);
}
// Shifts depth and site depth (a donor subtree moved under another parent).
__host__ __device__ __forceinline__ uint64_t w_shift(uint64_t w, int ddepth, int dsval) {
  const int d = w_depth(w) + ddepth, v = w_sval(w) + dsval;
  return (w & ~(0xffffULL << 32)) | (uint64_t(uint32_t(d) & 0xffu) << 32) | (uint64_t(uint32_t(v) & 0xffu) << 40);
}
// Replaces the site (entry and class) of a word by another word's site.
__host__ __device__ __forceinline__ uint64_t w_with_site(uint64_t w, uint64_t site_from) {
  const uint64_t mask = (0xffffULL << 16) | (0x7ffULL << 53);
  return (w & ~mask) | (site_from & mask);
}
__host__ __device__ __forceinline__ int len_nodes(int32_t l) { return l & 0xffff; }
__host__ __device__ __forceinline__ int len_consts(int32_t l) { return (l >> 16) & 0xffff; }
__host__ __device__ __forceinline__ int32_t make_len(int n, int c) { return n | (c << 16); }

// Definite assignment of grammar locals in a statement program
// (phase_locals_defined, cpp/src/evolution/repro/gpu/device/phase_compile.cuh:170-200):
// a grammar local may be read after an assignment to it, inside a for_range
// body that names it, and after a statement if only when both branches
// assigned it; a loop body's assignments do not outlive the loop, and inputs
// are always defined.  `at(i)` gives node i's tree kind, operand, arity and
// type.  False also for a tree deeper than 64 open nodes or one that ends
// early.
struct StatementNode {
  int kind, operand, arity, type;
};
// (`at` may be host-only: the engine's host code checks imported rows with it)
#pragma nv_exec_check_disable
template <class At>
__host__ __device__ inline bool locals_defined(int n, At at) {
  struct Frame {
    int16_t index, seen;
    uint16_t saved, branch;
  };
  Frame frames[64];
  int depth = 0;
  unsigned mask = 0;
  auto bit = [](int operand) -> unsigned { return operand >= 0 && operand < kNamedLocals ? 1u << operand : 0u; };
  for (int i = 0; i < n; ++i) {
    const StatementNode x = at(i);
    if (x.kind == TK_VAR && !(mask & bit(x.operand))) return false;
    if (x.arity > 0) {
      if (depth == 64) return false;
      frames[depth++] = Frame{int16_t(i), 0, uint16_t(mask), 0};
      continue;
    }
    while (depth) {
      Frame& f = frames[depth - 1];
      const StatementNode owner = at(f.index);
      ++f.seen;
      if (owner.kind == TK_FOR_RANGE && f.seen == 1) {
        f.saved = uint16_t(mask);
        mask |= bit(owner.operand);
      } else if (owner.kind == TK_IF && is_statement_tag(owner.type)) {
        if (f.seen == 1) {
          f.saved = uint16_t(mask);
        } else if (f.seen == 2) {
          f.branch = uint16_t(mask);
          mask = f.saved;
        } else {
          mask &= f.branch;
        }
      }
      if (f.seen < owner.arity) break;
      if (owner.kind == TK_ASSIGN) mask |= bit(owner.operand);
      else if (owner.kind == TK_FOR_RANGE) mask = f.saved;
      --depth;
    }
  }
  return depth == 0;
}

struct GenResult {
  int status, nodes, constants;
  int steps;  // tasks processed
};

// The subtree generator's tables: the sections of a search's GenImage, in
// shared memory (the variation kernel's staged copy) or in global memory.
// Read with plain loads, which serve either.
struct GenTables {
  const GenExpr* gx;
  const GenNt* gnt;
  const GenLevel* level;
  const GenEntry* entry;
  const GenDomain* doms;
  const gagp_value* vals;
  const uint32_t* cell;
  const uint16_t* row_of;
  const int4* extra;  // children 4..7 and their rows, two int4 per expression (arity above 4 only)
};
__device__ __forceinline__ GenTables gen_tables(const SearchDesc& s, const char* image) {
  return GenTables{reinterpret_cast<const GenExpr*>(image), reinterpret_cast<const GenNt*>(image + s.gi.nt),
                   reinterpret_cast<const GenLevel*>(image + s.gi.level),
                   reinterpret_cast<const GenEntry*>(image + s.gi.entry),
                   reinterpret_cast<const GenDomain*>(image + s.gi.doms),
                   reinterpret_cast<const gagp_value*>(image + s.gi.vals),
                   reinterpret_cast<const uint32_t*>(image + s.gi.cell),
                   reinterpret_cast<const uint16_t*>(image + s.gi.row_of),
                   reinterpret_cast<const int4*>(image + s.gi.extra)};
}

// The draws of one generator stream in order.  Warp: every lane takes the
// same draws, mixed 32 at a time (the stream is a counter mixed per draw); a
// draw is then one shuffle, started when the one before it is taken.
template <bool Warp>
struct DrawStream {
  Rng random;
  uint64_t ahead, batch = 0;
  int at = 0;
  __device__ __forceinline__ explicit DrawStream(uint64_t seed) : random(seed) { refill(); }
  __device__ __forceinline__ void refill() {
    if (Warp) {
      Rng mine(random.state + (threadIdx.x & 31) * 0x9e3779b97f4a7c15ULL);
      batch = mine.next();
      random.state += 32 * 0x9e3779b97f4a7c15ULL;
      at = 0;
      ahead = __shfl_sync(kFull, batch, 0);
    } else {
      ahead = random.next();
    }
  }
  __device__ __forceinline__ uint64_t next() {
    const uint64_t v = ahead;
    if (Warp && ++at < 32) ahead = __shfl_sync(kFull, batch, at);
    else refill();
    return v;
  }
};

// generate_phase<CompactTasks=true, EmitSites=true, Warp=false>
// (cpp/src/evolution/repro/gpu/device/phase_generate.cuh:125-270): a typed
// random subtree with min-cost feasibility and the FP64 weighted production
// draw.  The sequential draw uses round-to-nearest intrinsics so nothing is
// contracted into an FMA; the reference's host build rounds every operation
// alike.  Tasks pack (expression:17, depth:7, scope_count:4, logical:4) in
// `pending` (192 entries).  Emitted words carry depth relative to the generated
// root (root = 1) and site depth relative to the budget `logical_depth`.
//
// Warp: the warp generates one subtree, every lane with the same state (the
// lanes store the same words to the same addresses), and the lanes compare a
// draw with a production each; otherwise each thread generates its own.
//
// What bounds it: the chain of one subtree's steps, which sets the variation
// kernel's slowest child (an instruction every 5 cycles, most of them waiting
// for the one before).  A task carries what its cell holds (minimum cost, a
// reference's draw level), so a nonterminal and the production drawn for it
// are one step of four lookups: the level, the limits (a lane each, the choice
// value's FP64 multiplications and thresholds folded into 53-bit limits), the
// production and its children's cells.  Draws are mixed ahead and a constant's
// residue takes no division.  On the staged tables of the large scalar
// grammar, a warp alone takes 393 cycles per task (514 with every SM full); a
// lookup chain per task with the same draws took 637 (840).  The slowest
// child of a resumed search of P = 777 generated for 112k cycles with the
// draws in FP64 on one lane, 61k now.
template <bool Warp>
__device__ inline GenResult generate(const SearchDesc& s, const char* image, int root_expression, int scope_count,
                                     int depth, int capacity, uint64_t seed, uint64_t* out_node, int64_t* out_cval,
                                     int logical_depth, uint64_t* pending) {
  GenResult result{ST_INVALID, 0, 0, 0};
  const GenTables tables = gen_tables(s, image);
  const GenExpr* __restrict__ gx = tables.gx;
  const GenLevel* __restrict__ gen_level = tables.level;
  const GenEntry* __restrict__ gen_entry = tables.entry;
  const uint32_t* __restrict__ cell_words = tables.cell;
  const int n_ex = s.n_ex;
  const int depth_count = s.depth_count, logical_count = s.logical_count, cells = depth_count * logical_count;
  const int site_step = s.site_depth > 0 ? 1 : 0;
  if (root_expression < 0 || root_expression >= n_ex || scope_count < 0 || scope_count > 15 || depth <= 0 ||
      depth >= depth_count || depth > 64 || logical_depth < 0 || logical_depth >= logical_count ||
      capacity <= 0 || capacity > kCapacity || n_ex > 131071)
    return result;
  if (capacity > s.stride) capacity = s.stride;  // callers pass at most the node budget
  // A task: its cell word (its minimum cost, reserved when it was pushed, and
  // its level), and its expression with its depth (root 1) << 16 and the site
  // budget used << 24, as its node word holds them.  Scopes are not kept:
  // references are unscoped and nothing else asks.  The task to run next is
  // kept in registers rather than pushed and popped at once; `count` is what
  // the reference's stack holds below it.  What cannot happen with the tables
  // admission checks (a task that was not reserved, a full stack at a
  // nonterminal) is not tested, and a step's tests are one branch: every step
  // emits a node or ends, so the loop is bounded by the capacity.
  uint2* const stack = reinterpret_cast<uint2*>(pending);
  uint2* const words_out = reinterpret_cast<uint2*>(out_node);
  const int origin = (depth + 1) * logical_count + logical_depth;  // a node's cell is `origin` less its depth's and budget's
  uint2 task = make_uint2(cell_words[int(tables.row_of[root_expression]) * cells + depth * logical_count + logical_depth],
                          unsigned(root_expression) | 1u << 16);
  int count = 0;
  unsigned reserved = task.x & 0xffffu, room = unsigned(capacity);
  if (reserved > room) { result.status = ST_CAPACITY; return result; }
  DrawStream<Warp> random(seed);
  for (;;) {
    unsigned e = task.y & 0xffffu, place = task.y >> 16;
    unsigned site = 0, site_class = kNoClass << 21;
    const unsigned level = task.x >> 16;
    reserved -= task.x & 0xffffu;
    ++result.steps;
    if (level != kNoReference) {
      // a nonterminal and the production drawn for it, which runs at once.
      // Admission: the target nonterminal exists, is unscoped (as is every
      // reference) and its productions are in range.
      site = (e + 1) << 16;
      site_class = gx[e].shape << 21;
      place += unsigned(site_step) << 8;
      const unsigned available = room - reserved;
      // the widest precomputed level whose productions all fit: bound, first
      // entry, count, next narrower level
      int4 lv = *reinterpret_cast<const int4*>(gen_level + level);
      bool drawn = true;
      if (unsigned(lv.x) > available) {
        while (unsigned(lv.x) > available && lv.w >= 0) lv = *reinterpret_cast<const int4*>(gen_level + lv.w);
        drawn = unsigned(lv.x) <= available;
      }
      if (drawn) {
        const uint64_t bits = random.next() >> 11;
        const GenEntry* __restrict__ en = gen_entry + unsigned(lv.y);
        int pick = 0;
        if (Warp) {
          // lanes past the productions repeat the last one's limit
          const int last = lv.z - 1;
          int k = min(int(threadIdx.x & 31), last);
          unsigned hits = __ballot_sync(kFull, bits < en[k].limit);
          while (!hits) {  // the last feasible production's limit is past every draw
            pick += 32;
            k = min(pick + int(threadIdx.x & 31), last);
            hits = __ballot_sync(kFull, bits < en[k].limit || pick > last);
          }
          pick = min(pick + __ffs(hits) - 1, last);
        } else {
          while (pick < lv.z - 1 && bits >= en[pick].limit) ++pick;
        }
        e = unsigned(en[pick].expression);
      } else {
        // the reference's draw step by step (no precomputed level applies)
        const int budget = logical_depth - int(place >> 8), t_depth = depth + 1 - int(place & 0xffu);
        if (room == 0 || t_depth < 1 || budget < 0) { result.status = ST_CAPACITY; return result; }
        const int4 nt = *reinterpret_cast<const int4*>(tables.gnt + gx[e].target);
        const int nt_offset = nt.x;
        const bool normalized = nt.w != 0;
        const gagp_production* __restrict__ prods = s.prods;
        const uint32_t* __restrict__ prow = s.prod_minimum + (t_depth * logical_count + budget) * s.n_prods + nt_offset;
        uint64_t feasible_mask = 0;  // a bit per production for the first 64
        for (int i = 0; i < nt.y && i < 64; ++i)
          if (__ldg(&prow[i]) <= available) feasible_mask |= 1ULL << i;
        auto feasible = [&](int i) -> bool {
          return i < 64 ? (feasible_mask >> i & 1) : __ldg(&prow[i]) <= available;
        };
        double maximum = normalized ? 1.0 : 0.0, total = 0.0;
        if (!normalized)
          for (int i = 0; i < nt.y; ++i) {
            const double w = __ldg(&prods[nt_offset + i].weight);
            if (feasible(i) && w > maximum) maximum = w;
          }
        if (!(maximum > 0)) { result.status = ST_CAPACITY; return result; }
        for (int i = 0; i < nt.y; ++i)
          if (feasible(i)) {
            const double w = __ldg(&prods[nt_offset + i].weight);
            total = __dadd_rn(total, normalized ? w : __ddiv_rn(w, maximum));
          }
        double choice = __dmul_rn(__dmul_rn(double(random.next() >> 11), 0x1.0p-53), total);
        int production = -1;
        for (int i = 0; i < nt.y; ++i) {
          if (!feasible(i)) continue;
          production = __ldg(&prods[nt_offset + i].expression);
          const double w = __ldg(&prods[nt_offset + i].weight);
          choice = __dsub_rn(choice, normalized ? w : __ddiv_rn(w, maximum));
          if (choice < 0) break;
        }
        if (production < 0) return result;
        e = unsigned(production);
      }
      ++result.steps;
    }
    const int4 ra = *reinterpret_cast<const int4*>(gx + e);  // children, target, shape
    const unsigned shape = unsigned(ra.w), kind = shape >> 24, arity = shape >> 16 & 0xfu;
    const bool over = room == 0 || (place & 0xffu) > unsigned(depth) || place >> 8 > unsigned(logical_depth);
    if (over || kind == EK_REFERENCE || kind == EK_ALIAS) {
      // no room; a production that is a reference (a site within a site); an
      // alias (declined at admission)
      result.status = over && kind != EK_REFERENCE ? ST_CAPACITY : ST_INVALID;
      return result;
    }
    words_out[result.nodes++] = make_uint2(e | site, place | (shape & kShapeNode) | site_class);
    --room;
    if (arity == 0) {
      if (kind == EK_CONSTANT) {
        // admission: the domain exists and is an Int range or a list of Ints
        const GenDomain* dom = tables.doms + ra.z;
        uint64_t v = random.next();
        const uint64_t width = dom->width;
        if (width) {
          const uint64_t reject = dom->reject;
          while (v < reject) v = random.next();
          v -= __umul64hi(v, dom->magic) * width;  // at most two below the quotient
          v = v >= width ? v - width : v;
          v = v >= width ? v - width : v;
        }
        const int offset = dom->offset;
        out_cval[result.constants++] = offset < 0 ? int64_t(uint64_t(dom->minimum) + v) : tables.vals[offset + int(v)].i;
      }
      if (!count) break;
      task = stack[--count];
      continue;
    }
    // an operation: the children's minimum costs are reserved and the children
    // pushed last to first (the first straight into `task`); a step that
    // cannot reserve them all, or push past the stack, ends the generation
    const int4 rows = *(reinterpret_cast<const int4*>(gx + e) + 1);
    ++place;
    const uint32_t* __restrict__ words = cell_words + (origin - int(place & 0xffu) * logical_count - int(place >> 8));
    if (count + int(arity) - 1 >= 192 || (place & 0xffu) > unsigned(depth) + 1) {
      result.status = ST_CAPACITY;
      return result;
    }
    // kNoMinimum16 is past any room
    const uint32_t w0 = words[rows.x], w1 = arity > 1 ? words[rows.y] : 0u, w2 = arity > 2 ? words[rows.z] : 0u,
                   w3 = arity > 3 ? words[rows.w] : 0u;
    reserved += (w0 & 0xffffu) + (w1 & 0xffffu) + (w2 & 0xffffu) + (w3 & 0xffffu);
    const unsigned where = place << 16;
    if (arity > 4) {
      // a bounded region: children 4..7 from the image's extra section
      const int4 xa = tables.extra[2 * e], xb = tables.extra[2 * e + 1];
      for (int i = int(arity) - 1; i >= 4; --i) {
        const uint32_t word = words[i == 4 ? xb.x : i == 5 ? xb.y : i == 6 ? xb.z : xb.w];
        reserved += word & 0xffffu;
        stack[count++] = make_uint2(word, unsigned(i == 4 ? xa.x : i == 5 ? xa.y : i == 6 ? xa.z : xa.w) | where);
      }
    }
    if (reserved > room) { result.status = ST_CAPACITY; return result; }
    if (arity > 3) stack[count++] = make_uint2(w3, unsigned(ra.y) >> 16 | where);
    if (arity > 2) stack[count++] = make_uint2(w2, (unsigned(ra.y) & 0xffffu) | where);
    if (arity > 1) stack[count++] = make_uint2(w1, unsigned(ra.x) >> 16 | where);
    task = make_uint2(w0, (unsigned(ra.x) & 0xffffu) | where);
  }
  if (reserved || !result.nodes) return result;
  result.status = ST_OK;
  return result;
}

// ------------------------------------------------------- warp row primitives
// A row staged in shared memory: node words and constants.
struct SRow {
  uint64_t* node;
  int64_t* cval;
  int n, nc;
};

__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }

// site_matches (phase_operators.cuh:51-54): a variation site of class `cls`
// (any class when cls == kNoClass).
__device__ __forceinline__ bool site_matches(uint64_t w, uint32_t cls) {
  const uint32_t c = w_class(w);
  return c != kNoClass && (cls == kNoClass || c == cls);
}

// The position of set bit `rank` (from 0) of `mask`: the lane that many set
// bits lie below.  Every lane passes the same arguments.
__device__ __forceinline__ int warp_nth_bit(unsigned mask, unsigned rank) {
  const unsigned lane = lane_id();
  return __ffs(__ballot_sync(kFull, (mask >> lane & 1u) && unsigned(__popc(mask & ((1u << lane) - 1u))) == rank)) - 1;
}

// The variation sites of a row of at most 64 nodes (of class `cls`, of any when
// cls == kNoClass), kept so that a draw among them reads the row only once:
// crossover attempts draw from the same row again and again.
struct SiteSet {
  unsigned low, high;
  SmallRange range;
};
__device__ __forceinline__ SiteSet warp_sites(const SRow& t, uint32_t cls) {
  const int i = lane_id(), j = i + 32;
  const unsigned low = __ballot_sync(kFull, i < t.n && site_matches(t.node[i], cls));
  const unsigned high = __ballot_sync(kFull, j < t.n && site_matches(t.node[j], cls));
  return SiteSet{low, high, SmallRange(max(1u, unsigned(__popc(low) + __popc(high))))};
}
__device__ __forceinline__ int choose_site(const SiteSet& sites, Rng& random) {
  if (!(sites.low | sites.high)) return -1;
  const unsigned rank = random.bounded(sites.range), first = unsigned(__popc(sites.low));
  return rank < first ? warp_nth_bit(sites.low, rank) : 32 + warp_nth_bit(sites.high, rank - first);
}

// choose_site (phase_operators.cuh:55-83 and the counted warp variant
// :95-117): the same count, draws and prefix-ordered rank; reservoir draws
// visit matching sites in prefix order.  Every lane returns the same site.
// Out of line (a row of more than 64 nodes, or reservoir draws); returns the
// site (Drawn::value, -1 for none) and the stream's state.
__device__ __noinline__ Drawn choose_site_of(const uint64_t* node, int n, uint64_t state, bool counted, uint32_t cls) {
  const int lane = lane_id();
  Rng random(state);
  if (counted) {
    unsigned count = 0;
#pragma unroll 1
    for (int chunk = 0; chunk < n; chunk += 32) {
      const int i = chunk + lane;
      count += __popc(__ballot_sync(kFull, i < n && site_matches(node[i], cls)));
    }
    if (!count) return Drawn{~0ULL, random.state};
    unsigned rank = unsigned(random.bounded(count));
#pragma unroll 1
    for (int chunk = 0; chunk < n; chunk += 32) {
      const int i = chunk + lane;
      const unsigned mask = __ballot_sync(kFull, i < n && site_matches(node[i], cls));
      const unsigned c = __popc(mask);
      if (rank < c) return Drawn{uint64_t(chunk + warp_nth_bit(mask, rank)), random.state};
      rank -= c;
    }
    return Drawn{~0ULL, random.state};
  }
  int selected = -1;
  unsigned count = 0;
#pragma unroll 1
  for (int chunk = 0; chunk < n; chunk += 32) {
    const int i = chunk + lane;
    unsigned mask = __ballot_sync(kFull, i < n && site_matches(node[i], cls));
    while (mask) {
      const int bit = __ffs(mask) - 1;
      mask &= mask - 1;
      if (random.bounded(++count) == 0) selected = chunk + bit;
    }
  }
  return Drawn{uint64_t(int64_t(selected)), random.state};
}
__device__ __forceinline__ int warp_choose_site(const SRow& t, Rng& random, bool counted, uint32_t cls) {
  const Drawn d = choose_site_of(t.node, t.n, random.state, counted, cls);
  random.state = d.state;
  return int(int64_t(d.value));
}

// phase_subtree_end (device/phase_variation.cuh:81-91, warp form :213-229).
__device__ inline int warp_subtree_end(const SRow& t, int start) {
  // node words hold their depth: the subtree ends at the next node no deeper
  // than its root
  if (start < 0 || start >= t.n) return -1;
  const int lane = lane_id(), depth = w_depth(t.node[start]);
#pragma unroll 1
  for (int chunk = start + 1; chunk < t.n; chunk += 32) {
    const int i = chunk + lane;
    const unsigned hit = __ballot_sync(kFull, i < t.n && w_depth(t.node[i]) <= depth);
    if (hit) return chunk + __ffs(hit) - 1;
  }
  return t.n;
}

// Constant nodes among row positions [0, first) and [0, second), first <= second.
__device__ __forceinline__ void warp_count_constants2(const SRow& t, int first, int second, int* a, int* b) {
  int ca = 0, cb = 0;
#pragma unroll 1
  for (int chunk = 0; chunk < second; chunk += 32) {
    const int i = chunk + lane_id();
    const bool c = i < second && w_const(t.node[i]);
    ca += __popc(__ballot_sync(kFull, c && i < first));
    cb += __popc(__ballot_sync(kFull, c));
  }
  *a = ca;
  *b = cb;
}

// splice_phase_tree (device/phase_variation.cuh:147-207): base with the
// subtree [dest, end) replaced by donor's subtree [src, donor_end), into
// `out`; the callers have found both subtree ends already.
// Depth and site-depth limits are maxima of the output words; constants are
// base[..dest) ++ donor subtree ++ base[end..), the prefix renumbering the
// reference performs node by node.  Every lane returns the same result.
// `base_within`: base's own nodes are known to keep both limits, so only the
// donor's subtree is checked, before anything is written: most rejected
// splices are.
__device__ inline GenResult warp_splice(const SRow& base, bool base_within, int dest, int end, const SRow& donor, int src,
                                        int donor_end, SRow out, int stride, int max_depth, int site_limit) {
  GenResult r{ST_INVALID, 0, 0};
  if (max_depth <= 0 || max_depth > 64 || base.n <= 0 || donor.n <= 0 || dest < 0 || dest >= base.n || src < 0 ||
      src >= donor.n)
    return r;
  const uint64_t a = base.node[dest], b = donor.node[src];
  if (!w_site(a) || w_class(a) != w_class(b)) return r;
  if (end <= dest || end > base.n || donor_end <= src || donor_end > donor.n) return r;
  const int inserted = donor_end - src;
  const int length = base.n - (end - dest) + inserted;
  if (length > kCapacity) { r.status = ST_CAPACITY; return r; }
  if (length > stride) { r.status = ST_CAPACITY; return r; }  // never reached: callers bound by the node budget
  const int ddepth = w_depth(a) - w_depth(b), dsval = w_sval(a) - w_sval(b);
  int maxd = 0, maxs = 0;
#pragma unroll 1
  for (int i = src + lane_id(); i < donor_end; i += 32) {
    const uint64_t w = w_shift(donor.node[i], ddepth, dsval);
    maxd = max(maxd, w_depth(w));
    maxs = max(maxs, w_sval(w));
  }
  if (!base_within)
#pragma unroll 1
    for (int i = lane_id(); i < base.n; i += 32)
      if (i < dest || i >= end) {
        maxd = max(maxd, w_depth(base.node[i]));
        maxs = max(maxs, w_sval(base.node[i]));
      }
  if (__any_sync(kFull, maxd > max_depth || (site_limit && maxs > site_limit))) { r.status = ST_CAPACITY; return r; }
#pragma unroll 1
  for (int i = lane_id(); i < length; i += 32) {
    uint64_t w;
    if (i >= dest && i < dest + inserted) {
      w = w_shift(donor.node[src + i - dest], ddepth, dsval);
      if (i == dest) w = w_with_site(w, a);
    } else {
      w = base.node[i < dest ? i : i + (end - dest) - inserted];
    }
    out.node[i] = w;
  }
  int bb, be, db, de;
  warp_count_constants2(base, dest, end, &bb, &be);
  warp_count_constants2(donor, src, donor_end, &db, &de);
  const int dc = de - db;
#pragma unroll 1
  for (int k = lane_id(); k < bb; k += 32) out.cval[k] = base.cval[k];
#pragma unroll 1
  for (int k = lane_id(); k < dc; k += 32) out.cval[bb + k] = donor.cval[db + k];
#pragma unroll 1
  for (int k = lane_id(); k < base.nc - be; k += 32) out.cval[bb + dc + k] = base.cval[be + k];
  __syncwarp();
  r.status = ST_OK;
  r.nodes = length;
  r.constants = bb + dc + (base.nc - be);
  return r;
}

}  // namespace gb
