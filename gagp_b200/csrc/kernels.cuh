// Kernels of one resident steady-state round and of search start-up.
//
// Every kernel works on a batch of searches: `descs` holds one SearchDesc per
// search and per-item kernels map a flat index to (search, item) with the
// offsets array (items of search i are [off[i], off[i+1])).  A single search
// is a batch of one.  Per round (run_phase_population_steady,
// cpp/src/evolution/evolve.cpp:388-427):
//   k_record (epoch start) -> k_vary -> k_lower -> k_vm_fast / k_vm_exact / k_vm_region
//   -> k_place (k_place_cluster for large rounds) -> k_commit
#pragma once
#include <cooperative_groups.h>

#include "operators.cuh"
#include "accumulator.cuh"
#include "exact.cuh"

namespace gb {

namespace cg = cooperative_groups;

struct ProgramRef {
  int32_t search, slot;
};

__device__ __forceinline__ int find_search(const int32_t* off, int n, int item) {
  int lo = 0, hi = n;  // off[lo] <= item < off[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (off[mid] <= item) lo = mid; else hi = mid;
  }
  return lo;
}
__device__ __forceinline__ bool search_live(const SearchDesc& s) { return !s.round[2] && !s.round[3]; }
__device__ __forceinline__ void raise_error(const SearchDesc& s, int code) { atomicCAS(&s.round[3], 0, code); }

// ----------------------------------------------------------- start-up
// generate_phase_initial_population for a one-phase whole program
// (cpp/src/evolution/repro/gpu/phase_population_cpu.cpp:54-113): member i is
// grown at site depth 2 + i mod (site_depth - 1), retried with fresh seeds
// and raised by one every fourth failure.
__global__ void k_init_population(const SearchDesc* descs, const int32_t* off, int n) {
  const int item = blockIdx.x * blockDim.x + threadIdx.x;
  if (item >= off[n]) return;
  const int si = find_search(off, n, item);
  const SearchDesc& s = descs[si];
  if (s.imported) return;  // the caller's rows are the initial population
  const int i = item - off[si];
  const int site_limit = s.site_depth;
  const int ramp = site_limit < 2 ? site_limit : 2 + i % (site_limit - 1);
  uint64_t* node = s.node + size_t(i) * s.stride;
  int64_t* cval = s.cval + size_t(i) * s.stride;
  uint64_t pending[192];
  GenResult g{ST_INVALID, 0, 0, 0};
  for (int logical = ramp, attempt = 0; g.status != ST_OK; ++attempt) {
    const int room = s.maxv < kCapacity ? s.maxv : kCapacity;
    g = generate<false>(s, s.gen_image, s.root_expression, 0, s.slot_max_depth, room,
                 mix64(s.seed ^ mix64((uint64_t(i) * 8 + 0) * 64 + uint64_t(attempt))), node, cval, logical, pending);
    // a statement program that reads a grammar local before assigning it
    // is retried with the next seed (phase_population_cpu.cpp:95-96)
    if (g.status == ST_OK && is_statement_tag(s.slot_type) && !row_locals_defined(s, node, g.nodes))
      g.status = ST_INVALID;
    if (g.status != ST_OK && attempt % 4 == 3 && logical < site_limit) ++logical;
    if (attempt >= 256 && g.status != ST_OK) {
      raise_error(s, 20);
      s.len[i] = make_len(1, 0);
      return;
    }
  }
  // site depths relative to the budget `logical` are absolute here: the root
  // phase starts with no site above it
  s.len[i] = make_len(g.nodes, g.constants);
}

// Packed ranking key: (-fitness, wrong, nodes); smaller is better.
__device__ __forceinline__ uint64_t pack_key(const SearchDesc& s, double fitness, uint32_t wrong, uint32_t nodes) {
  const uint64_t loss = uint64_t(-fitness);
  if (!s.has_wrong) return loss;
  return (loss << s.key_shift_wrong) | (uint64_t(wrong) << s.key_shift_nodes) | uint64_t(nodes);
}

// A child that reuses member `source`'s result (an unchanged parent, an
// identical member): its statistics and key, by one lane.  The members'
// statistics stand until the round's commit.
__device__ inline void reuse_result(const SearchDesc& s, int b, int source) {
  s.c_fitness[b] = s.fitness[source];
  s.c_wrong[b] = s.wrong[source];
  s.c_nodes[b] = s.nodes[source];
  s.c_key[b] = s.key[source];
  atomicAdd(reinterpret_cast<unsigned long long*>(&s.counters[1]), 1ULL);
  // the generational evaluate copies a reused member's case counts too
  // (HostPhasePopulation::evaluate, phase_population_cpu.cpp:252-253), so
  // its program-case total covers every member
  if (s.generational) atomicAdd(reinterpret_cast<unsigned long long*>(&s.counters[2]), (unsigned long long)s.C);
}

// ----------------------------------------------------------- lowering
// Where lowered programs are listed, with each list's size: accumulator
// programs, register code, reference bytecode for the per-thread
// interpreter, and programs with bounded regions.
// Register code shares one list of `exact_capacity`: programs of at most
// kExactNarrow slots from its front, the others from its back.
struct LowerLists {
  ProgramRef *fast, *exact, *general, *region;
  int exact_capacity;
  int32_t *fast_count, *exact_count, *wide_count, *general_count, *region_count;
};
// mode 0: the members (initial evaluation); mode 1: this round's children
// that reuse no member's result; batch items [lo, hi).  One warp per row:
// the accumulator program when the row is total and fits the fuel, else
// register code for the exact VM, else the reference bytecode (lane 0).
// Exact false: no program of the batch can need the exact VM
// (exact_possible in vm_choice.cuh), so the other lowerings, with their shared
// memory and local arrays, stay out of the kernel and a row the accumulator
// lowering rejects is one the reference's compiler rejects too.
// Rows a block: a block's slowest row keeps its place, so without the exact
// lowerings one (a large scalar search 273 / 246 us per round with four rows,
// 266 / 241 with two, 264 / 240 with one); with them, whose local arrays make
// a block's start dear, two (list 341, 330 and 349 us).
template <bool Exact>
constexpr int kLowerWarps = Exact ? 2 : 1;
union LowerSmem {
  LowerScratch fast;
  ExactScratch exact;
};
template <bool Exact>
__global__ void __launch_bounds__(kLowerWarps<Exact> * 32, Exact ? 14 : 32)
    k_lower(const SearchDesc* descs, const int32_t* off, int n, int mode, LowerLists lists, int lo, int hi) {
  using Scratch = typename std::conditional<Exact, LowerSmem, LowerScratch>::type;
  __shared__ Scratch scratch[kLowerWarps<Exact>];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  LowerScratch& fast_scratch = reinterpret_cast<LowerScratch&>(scratch[warp]);
  const int total_items = min(off[n], hi);
  for (int item = lo + blockIdx.x * kLowerWarps<Exact> + warp; item < total_items;
       item += gridDim.x * kLowerWarps<Exact>) {
    const int si = find_search(off, n, item);
    const SearchDesc& s = descs[si];
    if (!search_live(s)) continue;
    const int slot = item - off[si];
    LRow t;
    if (mode == 0) {
      const int32_t l = s.len[slot];
      t = LRow{s.node + size_t(slot) * s.stride, s.cval + size_t(slot) * s.stride, len_nodes(l), len_consts(l)};
    } else {
      if (!s.c_eval[slot]) {
        if (lane == 0 && s.c_reuse[slot] >= 0) reuse_result(s, slot, s.c_reuse[slot]);
        continue;
      }
      const int32_t l = s.clen[slot];
      t = LRow{s.cnode + size_t(slot) * s.stride, s.ccval + size_t(slot) * s.stride, len_nodes(l), len_consts(l)};
      // a child its parent does not cover reuses an identical current
      // member's result when there is one (make_batch's member_hashes
      // lookup, phase_population_cpu.cpp:336-339) and is neither lowered
      // nor evaluated
      if (s.mtab) {
        const int m = warp_find_member(s, SRow{const_cast<uint64_t*>(t.node), const_cast<int64_t*>(t.cval), t.n, t.nc});
        if (m >= 0) {
          if (lane == 0) {
            s.c_reuse[slot] = m;
            s.c_eval[slot] = 0;
            reuse_result(s, slot, m);
          }
          continue;
        }
      }
    }
    int temps = 0;
    const int len = lower_accumulator_warp(s, t.node, t.n, t.cval, t.nc, s.code + size_t(slot) * s.code_stride,
                                           s.code_stride, s.kpool + size_t(slot) * s.stride, fast_scratch, &temps);
    // row and its length read; code words, constants, length, temps and list entry written
    const uint64_t row_bytes = 8ull * (t.n + t.nc) + 4;
    if (lane == 0) {
      s.vm_acc[2 * size_t(slot)] = 0;
      s.vm_acc[2 * size_t(slot) + 1] = 0;
      if (mode == 0 && s.errors) s.errors[slot] = 0;
    }
    if (len >= 0) {
      if (lane == 0) {
        s.code_len[slot] = len;
        s.code_temps[slot] = temps;
        lists.fast[atomicAdd(lists.fast_count, 1)] = ProgramRef{si, slot};
        atomicAdd(reinterpret_cast<unsigned long long*>(&s.counters[9]),
                  (unsigned long long)(row_bytes + 8ull * (len + t.nc) + 16));
      }
      continue;
    }
    if constexpr (!Exact) {
      if (lane == 0) raise_error(s, 30);  // the phase compiler rejects the row
    } else {
      int32_t* bc = s.bc + size_t(slot) * s.bc_pitch;
      int64_t* bc_consts = s.bc_consts + size_t(slot) * s.bc_stride;
      int slots = 0;
      int exact = kTooManySlots;
#pragma unroll 1
      for (int keep = 1; keep >= 0 && exact == kTooManySlots; --keep)
        exact = lower_exact_warp(s, t.node, t.n, t.cval, t.nc, reinterpret_cast<uint4*>(bc), s.bc_pitch / 4,
                                 bc_consts, scratch[warp].exact, keep, &slots);
      if (lane == 0) {
        if (exact >= 0) {
          const int at = slots <= kExactNarrow ? atomicAdd(lists.exact_count, 1)
                                               : lists.exact_capacity - 1 - atomicAdd(lists.wide_count, 1);
          lists.exact[at] = ProgramRef{si, slot};
          atomicAdd(reinterpret_cast<unsigned long long*>(&s.counters[9]),
                    (unsigned long long)(row_bytes + 16ull * (exact + 1) + 16));
        } else {
          LowerResult r{};
          const int bl = lower_program(lower_view(s), t.node, t.cval, t.n, t.nc, bc, s.bc_stride, bc_consts,
                                       s.bc_stride, &r);
          if (bl < 0) {
            raise_error(s, 30);  // the phase compiler rejected a constructed program
          } else {
            s.bc_len[slot] = bl;
            // the main code's length (a program with bounded regions: its
            // records and phase code follow); an exact-VM program keeps its
            // main constant count where an accumulator program keeps its
            // temporaries
            s.bc_locals[slot] = r.locals | (r.stack_bound << 8) | (r.main << 16);
            s.code_temps[slot] = r.main_constants;
            if (r.main < bl) lists.region[atomicAdd(lists.region_count, 1)] = ProgramRef{si, slot};
            else lists.general[atomicAdd(lists.general_count, 1)] = ProgramRef{si, slot};
            atomicAdd(reinterpret_cast<unsigned long long*>(&s.counters[9]),
                      (unsigned long long)(row_bytes + 20ull * bl + 8ull * r.constants + 16));
          }
        }
      }
      __syncwarp();
    }
  }
}

__device__ __forceinline__ void store_result(const SearchDesc& s, int mode, int slot, int64_t loss, uint32_t wrong) {
  const double f = -double(loss);
  const uint32_t w = s.has_wrong ? wrong : 0;
  if (mode == 0) {
    s.fitness[slot] = f;
    s.wrong[slot] = w;
  } else {
    // a child's ranking key too (evolve.cpp:403-413): with the reused
    // children's, formed as they are lowered, the placement reads keys only
    const uint32_t nodes = s.has_wrong ? ranking_nodes(s, s.cnode + size_t(slot) * s.stride, len_nodes(s.clen[slot])) : 0;
    s.c_fitness[slot] = f;
    s.c_wrong[slot] = w;
    s.c_nodes[slot] = nodes;
    s.c_key[slot] = pack_key(s, f, w, nodes);
  }
}

// One tile's loss and wrong count (and, where they are kept, its runtime
// errors) added to program `slot` of a search; returns whether this was the
// last of the program's `tiles` tiles, which then stores the program's
// result and counts its evaluation.  Loss (40 bits), wrong count (16) and
// finished tiles (8) share one word where they fit -- one atomic per tile
// and no fence -- and take two words with a fence between them otherwise.
// One lane calls it.
__device__ __forceinline__ bool add_tile_result(const SearchDesc& s, int mode, int slot, unsigned tiles, int64_t loss,
                                                uint32_t wrong, uint32_t errors) {
  unsigned long long* acc = s.vm_acc + 2 * size_t(slot);
  const uint64_t worst = s.metric == GAGP_METRIC_EXACT ? 1 : uint64_t(s.penalty_int);
  if (mode == 0 && s.errors && errors) atomicAdd(&s.errors[slot], errors);
  bool last;
  int64_t total;
  uint32_t total_wrong;
  if (tiles < 256 && s.C < 65536 && uint64_t(s.C) * worst < (1ULL << 40)) {
    const unsigned long long mine = (unsigned long long)loss | ((unsigned long long)wrong << 40) | (1ULL << 56);
    const unsigned long long sum = atomicAdd(&acc[0], mine) + mine;
    last = unsigned(sum >> 56) == tiles;
    total = int64_t(sum & ((1ULL << 40) - 1));
    total_wrong = uint32_t((sum >> 40) & 0xffffu);
  } else {
    atomicAdd(&acc[0], (unsigned long long)loss);
    __threadfence();
    const unsigned long long before = atomicAdd(&acc[1], (unsigned long long)wrong | (1ULL << 32));
    last = unsigned(before >> 32) == tiles - 1;
    total_wrong = uint32_t(before) + wrong;
    total = 0;
    if (last) {
      __threadfence();
      total = int64_t(atomicAdd(&acc[0], 0ULL));
    }
  }
  if (last) {
    store_result(s, mode, slot, total, total_wrong);
    atomicAdd(reinterpret_cast<unsigned long long*>(&s.counters[0]), 1ULL);
    atomicAdd(reinterpret_cast<unsigned long long*>(&s.counters[2]), (unsigned long long)s.C);
  }
  return last;
}

// The exact VMs: the programs the accumulator VM cannot run.  Persistent
// warps, each taking the next (program, tile of 32 cases) from `next`
// (zeroed before the launch): next[0] register code of few slots, next[1] of
// many, next[2] the interpreter's programs.  A tile adds its sums to the
// program's accumulators.
//
// Tiles are taken one warp at a time, not a block per program, because the
// tiles of a list program take unequal time (cases are ordered by list
// length): blocks spent half their warps' time at the barrier that ended a
// program.  All programs' last tiles, the longest lists, come first, so that
// the short ones fill the end of the launch.
//
// Dynamic shared memory per warp: kExactNarrow x 32 int64, and the code of a
// program of up to kExactStaged - 1 instructions (a longer one is read in
// place).  Programs of more slots run afterwards on every second warp, with
// the next warp's slots too.
constexpr int kExactWarps = 8, kExactBlocks = 4, kExactStaged = 64;
static_assert(kExactSlots == 2 * kExactNarrow, "a wide program takes two warps' slots");
constexpr size_t kExactSmem = size_t(kExactWarps) * (kExactNarrow * 32 * sizeof(int64_t) + kExactStaged * sizeof(uint4));
__device__ __noinline__ bool run_program_apart(const VmView& v, const int32_t* code, int n, const int64_t* consts,
                                               int n_locals, int c, int64_t* value, int* tag, uint64_t* steps) {
  return run_program(v, code, n, consts, n_locals, c, *value, *tag, *steps);
}
__global__ void __launch_bounds__(kExactWarps * 32, kExactBlocks) k_vm_exact(const SearchDesc* descs, int mode,
                                                                             LowerLists lists,
                                                                             unsigned long long* next, int max_C) {
  extern __shared__ __align__(16) int64_t smem_exact[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int64_t* slots = smem_exact + size_t(warp) * kExactNarrow * 32;
  uint4* staged = reinterpret_cast<uint4*>(smem_exact + size_t(kExactWarps) * kExactNarrow * 32) + warp * kExactStaged;
  const unsigned tiles_max = unsigned(max_C + 31) / 32;
  for (int which = 0; which < 3; ++which) {
    const unsigned count = unsigned(which == 0 ? *lists.exact_count : which == 1 ? *lists.wide_count : *lists.general_count);
    const unsigned long long items = (unsigned long long)count * tiles_max;
    if (which == 1) {
      if (!items) continue;
      __syncthreads();  // the narrow programs' slots are free
      if (warp & 1) continue;
    }
    for (;;) {
      if (!items) break;
      unsigned long long item = 0;
      if (lane == 0) item = atomicAdd(&next[which], 1ULL);
      item = __shfl_sync(kFull, item, 0);
      if (item >= items) break;
      const unsigned turn = items >> 32 ? unsigned(item / count) : unsigned(item) / count;
      const unsigned index = unsigned(item - (unsigned long long)turn * count);
      const ProgramRef p = which == 0   ? lists.exact[index]
                           : which == 1 ? lists.exact[lists.exact_capacity - 1 - int(index)]
                                        : lists.general[index];
      const SearchDesc& s = descs[p.search];
      const int c = int(tiles_max - 1 - turn) * 32 + lane;
      if (c - lane >= s.C) continue;
      const bool live = c < s.C;
      const VmView view = vm_view(s);
      const int32_t* code = s.bc + size_t(p.slot) * s.bc_pitch;
      const int64_t* consts = s.bc_consts + size_t(p.slot) * s.bc_stride;
      int64_t loss = 0;
      uint32_t wrong = 0, errors = 0;
      uint64_t steps = 0;
      bool ok = false;
      int64_t value = 0;
      int tag = s.result_type;
      if (which < 2) {
        const uint4* words = reinterpret_cast<const uint4*>(code);
        const uint4 head = __ldg(words);
        const int n = int(head.x & 0xffffu);
        const bool fits = n < kExactStaged;
        if (fits)
          for (int k = lane; k <= n; k += 32) staged[k] = __ldg(&words[1 + k]);
        __syncwarp();
        const ExactCase r = run_exact(view, fits ? staged : words + 1, head, consts, c, live, slots);
        __syncwarp();
        ok = r.ok;
        value = r.value;
        steps = r.steps;
      } else if (live) {
        ok = run_program_apart(view, code, s.bc_len[p.slot], consts, s.bc_locals[p.slot] & 0xff, c, &value, &tag, &steps);
      }
      if (live) {
        if (ok) loss = case_loss(s, tag, value, s.expected[c], wrong);
        else { loss = error_loss(s); wrong = 1; errors = 1; }
      }
      __syncwarp();
      loss = warp_sum(loss);
      wrong = warp_sum(wrong);
      errors = warp_sum(errors);
      steps = warp_sum(steps);
      if (lane == 0) {
        add_tile_result(s, mode, p.slot, unsigned((s.C + 31) / 32), loss, wrong, errors);
        atomicAdd(reinterpret_cast<unsigned long long*>(&s.counters[24]), (unsigned long long)steps);
      }
    }
  }
}

// Programs with bounded regions: a fixed grid of
// persistent warps, each taking the next (program, group of cases) from
// `next_item` (zeroed before the launch), one case per lane on the
// per-thread interpreter (run_program_regions), each lane with its own
// `ws_words` words of frames and memo cells in `ws` (`lanes` per warp).
//
// What bounds it: the cases of one program walk their recurrences along
// different paths, so lanes of a warp rarely share an instruction (2.7 of 32
// when a warp took 32 cases) and a warp's time is the sum of its lanes',
// while a round's few hundred programs left most of the GPU idle.  So a
// group is as small as still gives about kRegionItems items per warp: a
// round of 200 programs x 40 cases runs one case per warp.
constexpr int kRegionThreads = 128;
constexpr int kRegionItems = 4;
__global__ void __launch_bounds__(kRegionThreads) k_vm_region(const SearchDesc* descs, int mode, const ProgramRef* list,
                                                              const int32_t* list_count, unsigned long long* next_item,
                                                              int max_C, int lanes, int64_t* ws, size_t ws_words) {
  const int count = *list_count;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long warps = (long long)gridDim.x * (kRegionThreads / 32);
  int group = 1;
  while (group < lanes && (long long)count * max_C > kRegionItems * warps * group) group *= 2;
  const int groups = (max_C + group - 1) / group;
  const unsigned long long items = (unsigned long long)count * groups;
  int64_t* mine = ws + ((size_t(blockIdx.x) * (kRegionThreads / 32) + warp) * lanes + min(lane, lanes - 1)) * ws_words;
  for (;;) {
    unsigned long long item = 0;
    if (lane == 0) item = atomicAdd(next_item, 1ULL);
    item = __shfl_sync(kFull, item, 0);
    if (item >= items) break;
    const ProgramRef p = list[item / groups];
    const SearchDesc& s = descs[p.search];
    const int c = int(item % groups) * group + lane;
    if (c - lane >= s.C) continue;
    const int n = s.bc_len[p.slot], shape = s.bc_locals[p.slot];
    const int n_locals = shape & 0xff, n_main = (shape >> 16) & 0xffff;
    const int32_t* code = s.bc + size_t(p.slot) * s.bc_pitch;
    const int64_t* consts = s.bc_consts + size_t(p.slot) * s.bc_stride;
    const int main_consts = s.code_temps[p.slot];
    const VmView view = vm_view(s);
    int64_t loss = 0;
    uint32_t wrong = 0, errors = 0;
    uint64_t steps = 0;
    if (lane < group && c < s.C) {
      int64_t value = 0;
      int tag = 0;
      if (run_program_regions(view, s.regions, s.n_regions, code, n, n_main, consts, main_consts, n_locals, c, mine,
                              ws_words, value, tag, steps)) {
        loss += case_loss(s, tag, value, s.expected[c], wrong);
      } else {
        loss += error_loss(s);
        ++wrong;
        ++errors;
      }
    }
    __syncwarp();
    loss = warp_sum(loss);
    wrong = warp_sum(wrong);
    errors = warp_sum(errors);
    steps = warp_sum(steps);
    if (lane == 0) {
      add_tile_result(s, mode, p.slot, unsigned((s.C + group - 1) / group), loss, wrong, errors);
      atomicAdd(reinterpret_cast<unsigned long long*>(&s.counters[24]), (unsigned long long)steps);
    }
  }
}

// Fast VM: persistent warps over the fast list.  Per warp shared memory:
// temporaries (kMaxTemps x K x 32), the staged code (code_stride) and
// constants (stride).  Work items are (program, group of tiles of 32 K
// cases), program-major, so that a round with fewer programs than resident
// warps still fills the GPU; a group's tiles share the staging of the
// program, and groups grow while every warp keeps kVmItems items.  Each group
// adds its loss and wrong count to the program's accumulators and the last to
// finish stores the program's result (integer sums: the order does not
// matter).
// (Items a warp: 16384 programs on 2000 cases, a whole call: 8 1.54 ms, a warp
// of long programs runs on alone; 16 1.44; 32 1.46, every tile staged anew.)
constexpr int kVmItems = 16;
template <int K, int NIN>
__device__ __forceinline__ void run_group(const SearchDesc& s, int slot, const VmWarpSmem& w, const uint8_t* entries,
                                          int len, int case_begin, int case_end, int64_t& loss, uint32_t& wrong) {
  stage_program<K, NIN>(s, slot, w, entries, len);
  for (uint32_t c = case_begin; c < uint32_t(case_end); c += 32 * K)
    run_accumulator<K, NIN>(s, w, c, min(uint32_t(case_end), c + 32 * K), loss, wrong);
}
// One instantiation per cases-per-lane K (each with its own register
// budget); the engine's autotuner picks K per batch shape.
template <int K>
__global__ void __launch_bounds__(256, K == 4 ? 3 : 4) k_vm_fast(const SearchDesc* descs, int mode, const ProgramRef* list,
                                                 const int32_t* list_count, int temp_stride, int code_stride,
                                                 int const_stride, int tiles_max) {
  extern __shared__ __align__(16) int64_t smem_vm[];
  __shared__ uint8_t entries[kStageEntries];
  if (threadIdx.x < kStageEntries) entries[threadIdx.x] = uint8_t(stage_entry(threadIdx.x));
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int warps = blockDim.x >> 5;
  const size_t per_warp = size_t(temp_stride) + size_t(code_stride) + size_t(const_stride);  // int64 units
  int64_t* base = smem_vm + size_t(warp) * per_warp;
  const VmWarpSmem w{base, reinterpret_cast<uint2*>(base + temp_stride), base + temp_stride + code_stride};
  const long long count = *list_count, step = (long long)gridDim.x * warps;
  const int group = int(max(1LL, min((long long)tiles_max, count * tiles_max / (kVmItems * step))));  // tiles
  const int groups = (tiles_max + group - 1) / group;
  const long long cases = (long long)group * (32 * K);
  // the warp's items, first and then every `step` further on: program and
  // group counted along, for a 64-bit division per item cost more than staging
  const long long first = (long long)blockIdx.x * warps + warp;
  long long program = first / groups;
  int g = int(first % groups);
  const long long program_step = step / groups;
  const int g_step = int(step % groups);
  for (; program < count; program += program_step, g += g_step) {
    if (g >= groups) {
      g -= groups;
      if (++program >= count) break;
    }
    const ProgramRef p = list[program];
    const long long case0 = g * cases;
    const SearchDesc& s = descs[p.search];
    if (case0 >= s.C) continue;
    const int case1 = int(min((long long)s.C, case0 + cases));
    const int len = s.code_len[p.slot];
    int64_t loss = 0;
    uint32_t wrong = 0;
    switch (s.n_inputs) {
      case 1: run_group<K, 1>(s, p.slot, w, entries, len, int(case0), case1, loss, wrong); break;
      case 2: run_group<K, 2>(s, p.slot, w, entries, len, int(case0), case1, loss, wrong); break;
      default: run_group<K, 0>(s, p.slot, w, entries, len, int(case0), case1, loss, wrong); break;
    }
    loss = warp_sum(loss);
    wrong = warp_sum(wrong);
    if (lane == 0) {
      // accumulator programs never fail; the program's instructions over all
      // its cases are counted once
      if (add_tile_result(s, mode, p.slot, unsigned((s.C + cases - 1) / cases), loss, wrong, 0))
        atomicAdd(reinterpret_cast<unsigned long long*>(&s.counters[3]),
                  (unsigned long long)len * (unsigned long long)s.C);
    }
  }
}

// Member statistics after the initial evaluation.
__global__ void k_member_keys(const SearchDesc* descs, const int32_t* off, int n) {
  const int item = blockIdx.x * blockDim.x + threadIdx.x;
  if (item >= off[n]) return;
  const int si = find_search(off, n, item);
  const SearchDesc& s = descs[si];
  const int m = item - off[si];
  const uint32_t nodes = s.has_wrong ? ranking_nodes(s, s.node + size_t(m) * s.stride, len_nodes(s.len[m])) : 0;
  s.nodes[m] = nodes;
  s.key[m] = pack_key(s, s.fitness[m], s.wrong[m], nodes);
}

// ----------------------------------------------------------- run generator
// MT19937-64 (std::mt19937_64, evolve.cpp:339): the published Matsumoto-
// Nishimura generator.  The block regenerates the 312-word state in two
// dependency phases (words below 156 read only old words; words from 156 read
// the new word 156 positions back), tempers and appends the block.
__device__ __forceinline__ uint64_t mt_temper(uint64_t x) {
  x ^= (x >> 29) & 0x5555555555555555ULL;
  x ^= (x << 17) & 0x71D67FFFEDA60000ULL;
  x ^= (x << 37) & 0xFFF7EEE000000000ULL;
  x ^= x >> 43;
  return x;
}
__device__ __forceinline__ uint64_t mt_mix(uint64_t upper_src, uint64_t lower_src, uint64_t far) {
  const uint64_t x = (upper_src & 0xFFFFFFFF80000000ULL) | (lower_src & 0x7FFFFFFFULL);
  return far ^ (x >> 1) ^ ((x & 1) ? 0xB5026F5AA96619E9ULL : 0);
}
// x mod P from a multiply-high quotient estimate (Barrett): the estimate
// is at most two below floor(x / P), so at most two corrections follow.
__device__ __forceinline__ uint32_t mod_p(uint64_t x, uint64_t magic, uint32_t P) {
  const uint64_t q = __umul64hi(x, magic);
  uint64_t r = x - q * P;
  while (r >= P) r -= P;
  return uint32_t(r);
}
// Twists `mt` (smem, 312 words) using scratch `nw` (312 words) and appends
// the tempered block to the stream ring at stream position `wp`.
__device__ inline void mt_block(const SearchDesc& s, uint64_t* mt, uint64_t* nw, long long wp) {
  for (int i = threadIdx.x; i < 156; i += blockDim.x) nw[i] = mt_mix(mt[i], mt[i + 1], mt[i + 156]);
  __syncthreads();
  for (int i = 156 + threadIdx.x; i < 311; i += blockDim.x) nw[i] = mt_mix(mt[i], mt[i + 1], nw[i - 156]);
  __syncthreads();
  if (threadIdx.x == 0) nw[311] = mt_mix(mt[311], nw[0], nw[155]);
  __syncthreads();
  const int base = int(wp % s.stream_capacity);
  for (int i = threadIdx.x; i < 312; i += blockDim.x) {
    mt[i] = nw[i];
    const uint64_t out = mt_temper(nw[i]);
    int pos = base + i;
    if (pos >= s.stream_capacity) pos -= s.stream_capacity;
    s.stream[pos] = out;
    s.stream_mod[pos] = mod_p(out, s.mod_magic, uint32_t(s.P));
  }
  __syncthreads();
}
// Serial fallback of one block, for a consumer that ran ahead of the buffer.
__device__ inline void mt_block_serial(const SearchDesc& s, uint64_t* mt, long long wp) {
  for (int i = 0; i < 312; ++i) mt[i] = mt_mix(mt[i], mt[(i + 1) % 312], mt[(i + 156) % 312]);
  const int base = int(wp % s.stream_capacity);
  for (int i = 0; i < 312; ++i) {
    const uint64_t out = mt_temper(mt[i]);
    int pos = base + i;
    if (pos >= s.stream_capacity) pos -= s.stream_capacity;
    s.stream[pos] = out;
    s.stream_mod[pos] = mod_p(out, s.mod_magic, uint32_t(s.P));
  }
}

// stream_head as two 64-bit counters: [0] read, [1] written
__device__ __forceinline__ long long* stream_ptrs(const SearchDesc& s) { return s.stream_head; }

// Tops up each search's run-generator stream to the next placement's
// 2B+1 draws (as far as the ring allows).  Launched on a side stream so the
// generation overlaps the round's variation, lowering and evaluation; the
// placement kernel waits for it and only generates what redraws add.
//
// Thread t keeps words t and t + 156 of the state: the new ones need, besides
// the thread's own, only the next thread's old pair -- a shuffle, or shared
// memory at a warp's edge -- and the last thread, whose next words are the
// first thread's, forms word 0 itself.  One barrier per 312 outputs (three,
// with the state in shared memory, took 108 us for 32768 draws beside the
// variation, and the placement levels wait for them).
constexpr int kStreamThreads = 160;
__global__ void __launch_bounds__(kStreamThreads) k_stream(const SearchDesc* descs, int n) {
  __shared__ uint64_t edge_lo[2][kStreamThreads / 32], edge_hi[2][kStreamThreads / 32], second[2];
  const SearchDesc& s = descs[blockIdx.x];
  if (!search_live(s)) return;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const bool on = t < 156;
  uint64_t lo = on ? s.mt[t] : 0, hi = on ? s.mt[t + 156] : 0;
  const long long rp = stream_ptrs(s)[0];
  long long wp = stream_ptrs(s)[1];
  const long long need = (long long)s.B * s.replacement_size + 1;
  const int cap = s.stream_capacity;
  int at = int((wp + t) % cap);
  int buf = 0;
  __syncthreads();  // every thread has read the position
  while (wp - rp < need && wp - rp + 312 <= cap) {
    if (lane == 0) {
      edge_lo[buf][warp] = lo;
      edge_hi[buf][warp] = hi;
    }
    if (t == 1) second[buf] = lo;
    __syncthreads();
    uint64_t next_lo = __shfl_down_sync(kFull, lo, 1), next_hi = __shfl_down_sync(kFull, hi, 1);
    if (lane == 31 && warp + 1 < kStreamThreads / 32) {
      next_lo = edge_lo[buf][warp + 1];
      next_hi = edge_hi[buf][warp + 1];
    }
    if (t == 155) {
      next_lo = edge_hi[buf][0];
      next_hi = mt_mix(edge_lo[buf][0], second[buf], edge_hi[buf][0]);
    }
    lo = mt_mix(lo, next_lo, hi);
    hi = mt_mix(hi, next_hi, lo);
    if (on) {
      int far = at + 156;
      if (far >= cap) far -= cap;
      const uint64_t a = mt_temper(lo), b = mt_temper(hi);
      s.stream[at] = a;
      s.stream[far] = b;
      s.stream_mod[at] = mod_p(a, s.mod_magic, uint32_t(s.P));
      s.stream_mod[far] = mod_p(b, s.mod_magic, uint32_t(s.P));
    }
    at += 312;
    if (at >= cap) at -= cap;
    wp += 312;
    buf ^= 1;
  }
  if (on) {
    s.mt[t] = lo;
    s.mt[t + 156] = hi;
  }
  if (t == 0) stream_ptrs(s)[1] = wp;
}

// The `count` best members in ranking order (smallest (key, member) first),
// written to out[0..count): pass j takes the smallest (key, member) above
// pass j-1's.  For the generational schedule's elites this is the order of
// reproduce's stable sort by completed fitness (phase_population_cpu.cpp:
// 283-288): rank values when wrong counts are kept, fitness with ties to the
// lower index otherwise.  The whole block calls it; out[0] is the best.
__device__ inline void block_best_members(const SearchDesc& s, int count, int32_t* out) {
  __shared__ uint64_t top_key[32];
  __shared__ int top_idx[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = (blockDim.x + 31) >> 5;
  uint64_t prev_key = 0;
  int prev_idx = -1;
  for (int j = 0; j < count; ++j) {
    uint64_t bk = ~0ULL;
    int bi = 0x7fffffff;
    for (int m = threadIdx.x; m < s.P; m += blockDim.x) {
      const uint64_t k = s.key[m];
      const bool above = k > prev_key || (k == prev_key && m > prev_idx);
      if (above && (k < bk || (k == bk && m < bi))) { bk = k; bi = m; }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      const uint64_t k2 = __shfl_xor_sync(kFull, bk, o);
      const int i2 = __shfl_xor_sync(kFull, bi, o);
      if (k2 < bk || (k2 == bk && i2 < bi)) { bk = k2; bi = i2; }
    }
    if (lane == 0) { top_key[warp] = bk; top_idx[warp] = bi; }
    __syncthreads();
    bk = top_key[0];
    bi = top_idx[0];
    for (int w = 1; w < warps; ++w)
      if (top_key[w] < bk || (top_key[w] == bk && top_idx[w] < bi)) { bk = top_key[w]; bi = top_idx[w]; }
    __syncthreads();
    if (threadIdx.x == 0) out[j] = bi;
    prev_key = bk;
    prev_idx = bi;
  }
}

// Seeds the generator, tops up the stream, finds the best member and draws
// the first round's variation seed.  One block per search.
__global__ void k_start(const SearchDesc* descs, int n) {
  __shared__ uint64_t mt[312], nw[312];
  __shared__ uint64_t best_key[256];
  __shared__ int best_idx[256];
  const SearchDesc& s = descs[blockIdx.x];
  if (s.round[3]) return;
  if (threadIdx.x == 0) {
    mt[0] = s.seed;
    for (int i = 1; i < 312; ++i) mt[i] = 6364136223846793005ULL * (mt[i - 1] ^ (mt[i - 1] >> 62)) + uint64_t(i);
    stream_ptrs(s)[0] = 0;
    stream_ptrs(s)[1] = 0;
  }
  __syncthreads();
  mt_block(s, mt, nw, 0);
  // best member: smallest key, ties to the lowest index
  uint64_t bk = ~0ULL;
  int bi = 0x7fffffff;
  for (int m = threadIdx.x; m < s.P; m += blockDim.x) {
    const uint64_t k = s.key[m];
    if (k < bk || (k == bk && m < bi)) { bk = k; bi = m; }
  }
  best_key[threadIdx.x] = bk;
  best_idx[threadIdx.x] = bi;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int t = 1; t < blockDim.x; ++t)
      if (best_key[t] < bk || (best_key[t] == bk && best_idx[t] < bi)) { bk = best_key[t]; bi = best_idx[t]; }
    s.best[0] = bi;
    s.round_seed[0] = s.stream[0];  // the first run-generator output seeds round 0
    stream_ptrs(s)[0] = 1;
    stream_ptrs(s)[1] = 312;
    s.round[0] = 0;
    s.round[1] = 0;
    s.round[2] = s.total_rounds == 0;
  }
  for (int i = threadIdx.x; i < 312; i += blockDim.x) s.mt[i] = mt[i];
  if (s.generational && s.elite_count > 0) block_best_members(s, s.elite_count, s.elites);
}

// ----------------------------------------------------------- one round
// History entry before every population/batch rounds (record(),
// evolve.cpp:360-371): the best member, its row, and the exact integer sum of
// member fitness (the host forms the long double mean).
__global__ void __launch_bounds__(1024) k_record(const SearchDesc* descs, int n, int only_epoch_start) {
  __shared__ long long partial[1024];
  const SearchDesc& s = descs[blockIdx.x];
  if (!search_live(s)) return;
  const int round = s.round[0];
  if (only_epoch_start && round % s.rounds_per_epoch) return;
  const int entry = s.round[1];
  if (entry >= s.generations) return;
  long long sum = 0;
#pragma unroll 4
  for (int m = threadIdx.x; m < s.P; m += blockDim.x) sum += (long long)s.fitness[m];
  partial[threadIdx.x] = sum;
  __syncthreads();
  for (int w = blockDim.x / 2; w; w >>= 1) {
    if (threadIdx.x < w) partial[threadIdx.x] += partial[threadIdx.x + w];
    __syncthreads();
  }
  const int b = s.best[0];
  const int32_t l = s.len[b];
  for (int i = threadIdx.x; i < len_nodes(l); i += blockDim.x)
    s.hist_node[size_t(entry) * s.stride + i] = s.node[size_t(b) * s.stride + i];
  for (int i = threadIdx.x; i < len_consts(l); i += blockDim.x)
    s.hist_cval[size_t(entry) * s.stride + i] = s.cval[size_t(b) * s.stride + i];
  if (threadIdx.x == 0) {
    s.hist_sum[entry] = partial[0];
    s.hist_fitness[entry] = s.fitness[b];
    s.hist_wrong[entry] = s.wrong[b];
    s.hist_nodes[entry] = uint32_t(s.fixed_nodes + len_nodes(l));
    s.hist_len[entry] = l;
    s.round[1] = entry + 1;
  }
}

// The round's member index (HostPhasePopulation's member_hashes, kept
// current by commit_batch, phase_population_cpu.cpp:318-321,382-394): a warp
// per member hashes its row and inserts it by linear probing unless an
// identical row is indexed already, so every distinct row has one entry and
// the probe runs stay short however many copies the population holds.  A
// slot word carries the hash's top bits with the member, so a warp that
// loses a slot to another compares tags and then rows (stable in memory
// all round) without waiting for any other write.  At most P entries in at
// least 2P slots: every probe sequence meets an empty slot.  k_commit clears
// the table for the next round.
__global__ void __launch_bounds__(256) k_member_index(const SearchDesc* descs, const int32_t* off, int n) {
  const int item = int((size_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (item >= off[n]) return;
  const int si = find_search(off, n, item);
  const SearchDesc& s = descs[si];
  if (!search_live(s) || !s.mtab) return;
  const int m = item - off[si];
  const int32_t l = s.len[m];
  const uint64_t* node = s.node + size_t(m) * s.stride;
  const int64_t* cval = s.cval + size_t(m) * s.stride;
  const uint64_t h = warp_row_hash(node, cval, len_nodes(l), len_consts(l));
  const unsigned long long mine = index_word(h, m);
  const uint32_t mask = uint32_t(s.mtab_mask);
  uint32_t slot = uint32_t(h) & mask;
  for (uint32_t probe = 0; probe <= mask; ++probe) {
    unsigned long long cur = 0;
    if (lane == 0) cur = atomicCAS(&s.mtab[slot], 0ULL, mine);
    cur = __shfl_sync(kFull, cur, 0);
    if (!cur) return;  // indexed
    if (index_tag_matches(cur, h)) {
      const int other = index_member(cur);
      const int32_t lc = s.len[other];
      if (warp_rows_equal(s.node + size_t(other) * s.stride, s.cval + size_t(other) * s.stride, len_nodes(lc),
                          len_consts(lc), node, cval, len_nodes(l), len_consts(l)))
        return;  // an identical row is indexed already
    }
    slot = (slot + 1) & mask;
  }
}

// make_batch (phase_population_cpu.cpp:322-353): one warp per child, rows
// staged in dynamic shared memory (warp_rows_bytes(stride) per warp).
// Persistent warps over the batch items [lo, hi): each warp takes the next
// child from `next_item` (zeroed before the launch) until the range is
// varied, so warps that drew short children go on to the next one instead
// of idling.  When the range's children all belong to search `staged`, the
// block first copies that search's generator image (image_bytes) into
// shared memory after the rows: a generation step is a chain of dependent
// table lookups, each a shared-memory load instead of a global one.
// Bound by latency, of instruction fetches first: its warps are each somewhere
// else in 130 KB of code (4.7 of the 12 cycles an instruction waits, with 24
// warps an SM), so loops over a row's nodes are not unrolled and rare draws
// are out of line (174 KB before).  Five blocks an SM and 96 registers: six
// spill 200 bytes a thread, four are no faster (large scalar search 274 / 250
// us per round, generational 165 / 176; six 273 / 247 and 173 / 186).
__global__ void __launch_bounds__(128, 5) k_vary(const SearchDesc* descs, const int32_t* off, int n, int stride_max,
                                                 int32_t* next_item, int lo, int hi, int collect_stats, int staged,
                                                 int image_bytes) {
  extern __shared__ __align__(16) char smem_rows[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  char* base = smem_rows + size_t(warp) * warp_rows_bytes(stride_max);
  char* image = smem_rows + size_t(blockDim.x >> 5) * warp_rows_bytes(stride_max);
  if (staged >= 0) {
    const uint4* from = reinterpret_cast<const uint4*>(descs[staged].gen_image);
    uint4* to = reinterpret_cast<uint4*>(image);
    for (int i = threadIdx.x; i < image_bytes / 16; i += blockDim.x) to[i] = from[i];
    __syncthreads();
  }
  const int total = min(off[n], hi);
  for (;;) {
    int item = 0;
    if (lane == 0) item = lo + atomicAdd(next_item, 1);
    item = __shfl_sync(kFull, item, 0);
    if (item >= total) break;
    const int si = find_search(off, n, item);
    const SearchDesc& s = descs[si];
    if (!search_live(s)) continue;
    const int child = item - off[si];
    WarpRows rows = carve_rows(base, s.stride);
    int reuse = -1, parent = -1;
    long long stamp[5] = {0, 0, 0, 0, 0};
    const long long started = clock64();
    const int error = warp_vary_child(s, image, si == staged, child, s.round_seed[0], rows, &reuse, &parent, stamp);
    if (lane == 0 && collect_stats) {
      // per-phase SM cycles: selection, crossover, subtree generation, rest
      stamp[3] = clock64();
      long long prev = started;
      for (int k = 0; k < 4; ++k) {
        if (stamp[k] == 0) stamp[k] = prev;
        atomicAdd(reinterpret_cast<unsigned long long*>(&s.counters[10 + k]), (unsigned long long)(stamp[k] - prev));
        atomicMax(reinterpret_cast<unsigned long long*>(&s.counters[16 + k]), (unsigned long long)(stamp[k] - prev));
        prev = stamp[k];
      }
      atomicMax(reinterpret_cast<unsigned long long*>(&s.counters[15]), (unsigned long long)(stamp[3] - started));
      if (stamp[3] - started > 200000) atomicAdd(reinterpret_cast<unsigned long long*>(&s.counters[20]), 1ULL);
      if (stamp[4]) {
        atomicAdd(reinterpret_cast<unsigned long long*>(&s.counters[21]), (unsigned long long)(stamp[4] - 1));
        atomicMax(reinterpret_cast<unsigned long long*>(&s.counters[22]), (unsigned long long)(stamp[4] - 1));
        atomicAdd(reinterpret_cast<unsigned long long*>(&s.counters[23]), 1ULL);
      }
      // rows read (parent, donor) and written (child) with their lengths,
      // 2 x pressure tournament keys, four per-child outputs
      const uint64_t bytes = 8ull * (rows.parent.n + rows.parent.nc + rows.donor.n + rows.donor.nc + rows.child.n +
                                     rows.child.nc + 2 * s.pressure) + 12 + 16;
      atomicAdd(reinterpret_cast<unsigned long long*>(&s.counters[8]), (unsigned long long)bytes);
    }
    if (lane == 0) {
      s.c_parent[child] = parent;
      s.c_reuse[child] = reuse;
      s.c_error[child] = error;
      s.c_eval[child] = error == 0 && reuse < 0;
      if (error) raise_error(s, 100 + error);
    }
    __syncwarp();
  }
}

// State of every search of a batch in one array (bit 0: finished, bit 1:
// failed), so that a serving step reads them with one copy.
__global__ void k_status(const SearchDesc* descs, int n, int32_t* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const SearchDesc& s = descs[i];
  out[i] = (s.round[2] ? 1 : 0) | (s.round[3] ? 2 : 0);
}

// Shape of the cluster that finds a large round's placement levels
// (k_place_levels): kPlaceCtas blocks of kClusterThreads threads, kClusterPer
// children per thread.  Rounds that one block holds take one
// (k_place_levels_small).
constexpr int kPlaceCtas = 8;
constexpr int kClusterThreads = 1024;
constexpr int kClusterPer = 2;
constexpr int kLevelsSmall = kClusterThreads * kClusterPer;  // children
constexpr int kClusterMinChildren = 4096;  // rounds the cluster places (k_place_cluster)

// Windowed placement step over lanes [seg_begin, seg_end) of a window whose
// children's draws do not overlap (every lane's members differ from every
// earlier active lane's): victims from the current keys equal the
// sequential ones, the best member before each lane is an exclusive prefix
// minimum of (key, member), and the lanes commit up to the first whose
// victim is the current best (a redraw).  Returns the committed count.
__device__ __forceinline__ int place_segment(uint64_t* keys, int32_t* placed, int b0, int seg_begin, int seg_end,
                                             int d0, int d1, uint64_t ck, int& best, uint64_t& best_key) {
  const int lane = threadIdx.x & 31;
  const bool live = lane >= seg_begin && lane < seg_end;
  const uint64_t k0 = live ? keys[d0] : 0, k1 = live ? keys[d1] : 0;
  // worst of the pair: the second replaces the first when the first is better
  const int v = (k0 < k1 || (k0 == k1 && d0 < d1)) ? d1 : d0;
  uint64_t pk = live ? ck : ~0ULL;
  int pv = live ? v : 0x7fffffff;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint64_t uk = __shfl_up_sync(kFull, pk, o);
    const int uv = __shfl_up_sync(kFull, pv, o);
    if (lane >= o && (uk < pk || (uk == pk && uv < pv))) { pk = uk; pv = uv; }
  }
  uint64_t ek = __shfl_up_sync(kFull, pk, 1);
  int ev = __shfl_up_sync(kFull, pv, 1);
  if (lane == 0 || best_key < ek || (best_key == ek && best < ev)) { ek = best_key; ev = best; }
  const unsigned rmask = __ballot_sync(kFull, live && v == ev);
  const int stop = rmask ? __ffs(rmask) - 1 : seg_end;
  const int valid = stop - seg_begin;
  if (valid <= 0) return 0;
  if (live && lane < stop) {
    keys[v] = ck;
    placed[v] = b0 + lane;
  }
  uint64_t nk = __shfl_sync(kFull, pk, stop - 1);
  int nv = __shfl_sync(kFull, pv, stop - 1);
  if (best_key < nk || (best_key == nk && best < nv)) { nk = best_key; nv = best; }
  best_key = nk;
  best = nv;
  __syncwarp();
  return valid;
}

// Lanes of a 32-child window whose draws overlap an earlier lane's: bit j
// set when child j draws a member that some child i < j of the window drew.
__device__ __forceinline__ int latest_overlap(int d0, int d1) {
  const int lane = threadIdx.x & 31;
  int latest = -1;
#pragma unroll 8
  for (int o = 1; o < 32; ++o) {
    const int e0 = __shfl_up_sync(kFull, d0, o), e1 = __shfl_up_sync(kFull, d1, o);
    if (lane >= o && ((e0 == d0) | (e0 == d1) | (e1 == d0) | (e1 == d1))) latest = max(latest, lane - o);
  }
  return latest;
}

// Steady-state placement (evolve.cpp:414-427): children in order, each
// replacing the worst of replacement_size uniform draws (redrawn when it is
// the current best).  One block per search; `dyn_bytes`: dynamic shared
// memory of the launch (member keys, then the level owners or staged draws).
//
// Level-parallel path (replacement size 2): without a redraw child j draws
// stream positions 2j and 2j+1, and its level follows from the draws alone: a
// child is ready once it is the earliest unplaced child drawing each of its
// members (k_place_levels, run beside the variation).  The ready children of
// a level draw disjoint members, so they read exactly the keys the sequential
// loop would and place at once.  The best member before each child is then a
// prefix minimum of (key, member) in child order; a child whose victim is
// that best member would have redrawn (both its draws are the best member),
// and then the round is replayed on the exact windowed path.
//
// Windowed path (warp 0): 32 children per step, one per lane, over draws
// staged in shared memory; a step commits the lanes before the first lane
// drawing a member an earlier lane drew, or before the first redraw, which
// the sequential loop then takes.  Other replacement sizes and the end of
// the staged draws run the sequential loop.
// Finally the next round's seed is drawn.
constexpr int kPlaceThreads = 1024;
__device__ __forceinline__ bool key_before(uint64_t ka, int va, uint64_t kb, int vb) {
  return ka < kb || (ka == kb && va < vb);
}
// Per: children per thread of the level-parallel path, the fewest that hold
// the search's round (1 up to 1024 children, 4 up to 4096; past that the
// cluster places).  Bound by latency: a barrier and two shared-memory keys per
// level, some 11 levels.  Finding the levels here with two atomics and two
// barriers each, and copying the placed members' statistics (k_commit does),
// took a round of 1024 children 15 us and one of 2048 31, 9 and 14 now.
// With 16 children a thread for larger rounds, a child's key had to come from
// global memory each time: 88 us for 16384 against the cluster's 36.
struct PlaceShared {
  uint64_t mt[312], nw[312];
  uint64_t ck_stage[1024];
  uint64_t scan_key[32];
  int scan_idx[32];
  long long pos, wp;
  int best, fail, redraw_at;
};
// Whether a round of search s has placement levels: replacement size 2 and
// the whole round's draws in the stream.
__device__ __forceinline__ bool levels_apply(const SearchDesc& s, long long rp, long long wp) {
  return s.replacement_size == 2 && s.B <= kPlaceCtas * kClusterThreads * kClusterPer && wp - rp >= 2LL * s.B + 1;
}
template <int Per>
__device__ __noinline__ void place_round(const SearchDesc& s, PlaceShared& sh, uint64_t* keys, int dyn_bytes,
                                         bool replay) {
  uint64_t (&mt)[312] = sh.mt, (&nw)[312] = sh.nw, (&ck_stage)[1024] = sh.ck_stage, (&scan_key)[32] = sh.scan_key;
  int (&scan_idx)[32] = sh.scan_idx;
  long long &shared_pos = sh.pos, &shared_wp = sh.wp;
  int &shared_best = sh.best, &shared_fail = sh.fail, &redraw_at = sh.redraw_at;
  const long long t0 = clock64();
  const int P = s.P, B = s.B, rs = s.replacement_size, cap = s.stream_capacity;
  const int tid = threadIdx.x;
  int32_t* __restrict__ placed = s.placed;
  for (int m = tid; m < P; m += blockDim.x) keys[m] = s.key[m];
  for (int i = tid; i < 312; i += blockDim.x) mt[i] = s.mt[i];
  __syncthreads();
  static_assert(Per == 1 || Per == 4, "draws and levels are read in pairs and fours");
  uint64_t kept[Per];  // the children's keys
#pragma unroll
  for (int t = 0; t < Per; ++t) kept[t] = tid * Per + t < B ? s.c_key[tid * Per + t] : ~0ULL;
  const long long rp = stream_ptrs(s)[0];
  long long wp = stream_ptrs(s)[1];
  const long long need = (long long)B * rs + 1;
  while (wp - rp < need && wp - rp + 312 <= cap) {
    mt_block(s, mt, nw, wp);
    wp += 312;
  }
  const long long t1 = clock64();
  // ---------------------------------------------------- level-parallel path
  // after the keys, 16-byte aligned: first the staged draws, with 64 bytes
  // of slack for the per-thread 16-byte reads of them, then the child placed
  // on each member
  uint16_t* const stage = reinterpret_cast<uint16_t*>(keys + P + (P & 1));
  int16_t* const on = reinterpret_cast<int16_t*>(stage);
  const int after = dyn_bytes - int(sizeof(uint64_t)) * (P + 1) - 64;
  const bool parallel_path = !replay && levels_apply(s, rp, wp) && s.level_plan[0] == s.round[0] + 1 &&
                             blockDim.x == kPlaceThreads && B <= kPlaceThreads * Per &&
                             after >= int(sizeof(int16_t)) * max(P, 2 * B);
  bool parallel_done = false;
  if (parallel_path) {
    // thread tid owns children [Per tid, Per tid + Per): cand[t] holds child
    // begin + t's two draws, and once it is placed, its victim
    const int base = int(rp % cap);
    const int begin = tid * Per;
    // the 2B draws (residues < P <= 65536), staged as 16-bit values with
    // coalesced loads, then read back per thread: child j's pair is the
    // 32-bit word j
    {
      const uint32_t* __restrict__ smod = s.stream_mod;
      for (int i = tid; i < 2 * B; i += blockDim.x) {
        int pos = base + i;
        if (pos >= cap) pos -= cap;
        stage[i] = uint16_t(smod[pos]);
      }
    }
    // the children's levels, two a word (rows of child_level are padded)
    uint32_t level_pair[(Per + 1) / 2];
    if constexpr (Per == 1) {
      level_pair[0] = begin < B ? uint32_t(uint16_t(s.child_level[begin])) : 0xffffu;
    } else {
      const uint2 v = begin < B ? *reinterpret_cast<const uint2*>(s.child_level + begin) : make_uint2(~0u, ~0u);
      level_pair[0] = v.x;
      level_pair[1] = v.y;
    }
    __syncthreads();
    uint32_t cand[Per];
    {
      const uint32_t* words = reinterpret_cast<const uint32_t*>(stage);
      if constexpr (Per == 1) {
        cand[0] = begin < B ? words[begin] : 0;
      } else {
        const uint4 v = begin < B ? *reinterpret_cast<const uint4*>(words + begin) : make_uint4(0, 0, 0, 0);
        cand[0] = v.x;
        cand[1] = v.y;
        cand[2] = v.z;
        cand[3] = v.w;
      }
#pragma unroll
      for (int t = 0; t < Per; ++t)
        if (begin + t >= B) {
          cand[t] = 0;
          level_pair[t / 2] |= 0xffffu << (16 * (t & 1));  // no level
        }
    }
    __syncthreads();  // the staged draws give way to the placed children
    for (int m = tid; m < P; m += blockDim.x) on[m] = -1;
    if (tid == 0) redraw_at = 0x7fffffff;
    __syncthreads();
    const int levels_run = s.level_plan[1];
    const long long level_start = clock64();
    for (int level = 0; level < levels_run; ++level) {
#pragma unroll
      for (int t = 0; t < Per; ++t)
        if ((level_pair[t / 2] >> (16 * (t & 1)) & 0xffffu) == uint32_t(level)) {
          const int d0 = int(cand[t] & 0xffff), d1 = int(cand[t] >> 16);
          const uint64_t k0 = keys[d0], k1 = keys[d1];
          // worst of the pair: the second replaces the first when the first is better
          const int v = (k0 < k1 || (k0 == k1 && d0 < d1)) ? d1 : d0;
          keys[v] = kept[t];
          on[v] = int16_t(begin + t);
          cand[t] = uint32_t(v);
        }
      __syncthreads();
    }
    if (tid == 0)
      atomicAdd(reinterpret_cast<unsigned long long*>(&s.counters[14]), (unsigned long long)(clock64() - level_start));
    // best member before each child (child order): each thread's minimum of
    // (key, victim) over its children, a warp-shuffle scan, then a scan of
    // the warp totals, gives each thread's incoming best
    const int lane = tid & 31, warp = tid >> 5;
    uint64_t mk = ~0ULL;
    int mv = 0x7fffffff;
#pragma unroll
    for (int t = 0; t < Per; ++t)
      if (begin + t < B && key_before(kept[t], int(cand[t]), mk, mv)) {
        mk = kept[t];
        mv = int(cand[t]);
      }
    for (int o = 1; o < 32; o <<= 1) {
      const uint64_t uk = __shfl_up_sync(kFull, mk, o);
      const int uv = __shfl_up_sync(kFull, mv, o);
      if (lane >= o && key_before(uk, uv, mk, mv)) { mk = uk; mv = uv; }
    }
    constexpr int kWarps = kPlaceThreads / 32;
    if (lane == 31) { scan_key[warp] = mk; scan_idx[warp] = mv; }
    __syncthreads();
    if (warp == 0) {
      uint64_t wk = lane < kWarps ? scan_key[lane] : ~0ULL;
      int wv = lane < kWarps ? scan_idx[lane] : 0x7fffffff;
      for (int o = 1; o < 32; o <<= 1) {
        const uint64_t uk = __shfl_up_sync(kFull, wk, o);
        const int uv = __shfl_up_sync(kFull, wv, o);
        if (lane >= o && key_before(uk, uv, wk, wv)) { wk = uk; wv = uv; }
      }
      scan_key[lane] = wk;
      scan_idx[lane] = wv;
    }
    __syncthreads();
    const int best0 = s.best[0];
    const uint64_t best0_key = s.key[best0];
    int bv = best0;
    uint64_t bk = best0_key;
    {
      const uint64_t lk = __shfl_up_sync(kFull, mk, 1);
      const int lv = __shfl_up_sync(kFull, mv, 1);
      if (lane > 0 && key_before(lk, lv, bk, bv)) { bk = lk; bv = lv; }
      if (warp > 0 && key_before(scan_key[warp - 1], scan_idx[warp - 1], bk, bv)) {
        bk = scan_key[warp - 1];
        bv = scan_idx[warp - 1];
      }
    }
    // a child whose victim is the best member before it would have redrawn
    bool hit = false;
#pragma unroll
    for (int t = 0; t < Per; ++t)
      if (!hit && begin + t < B) {
        const int v = int(cand[t]);
        if (v == bv) {
          atomicMin(&redraw_at, begin + t);
          hit = true;
        } else if (key_before(kept[t], v, bk, bv)) {
          bk = kept[t];
          bv = v;
        }
      }
    __syncthreads();
    parallel_done = redraw_at == 0x7fffffff;
    if (tid == 0)  // levels of the parallel path; a replay adds 2^20
      atomicAdd(reinterpret_cast<unsigned long long*>(&s.counters[7]),
                (unsigned long long)levels_run + (parallel_done ? 0ULL : (1ULL << 20)));
    if (parallel_done) {
      if (tid == 0) {
        int fv = best0;
        uint64_t fk = best0_key;
        if (key_before(scan_key[kWarps - 1], scan_idx[kWarps - 1], fk, fv)) {
          fk = scan_key[kWarps - 1];
          fv = scan_idx[kWarps - 1];
        }
        shared_best = fv;
        shared_fail = 0;
        // the next round's seed: the raw output after the 2B placement draws
        const long long pos = rp + 2LL * B;
        s.round_seed[0] = s.stream[pos % cap];
        shared_pos = pos + 1;
        shared_wp = wp;
      }
      for (int m = tid; m < P; m += blockDim.x) placed[m] = on[m];
    } else {
      // replay the round on the exact windowed path from the round's keys
      for (int m = tid; m < P; m += blockDim.x) keys[m] = s.key[m];
    }
    __syncthreads();
  }
  if (!parallel_done)
    for (int m = tid; m < P; m += blockDim.x) placed[m] = -1;
  // ---------------------------------------------------- windowed path
  uint16_t* draws = reinterpret_cast<uint16_t*>(keys + P);
  const int slots = (dyn_bytes - int(sizeof(uint64_t)) * P) / int(sizeof(uint16_t));
  const int avail = int(min((long long)slots, wp - rp));
  if (!parallel_done) {
    const int base = int(rp % cap);
    for (int i = tid; i < avail; i += blockDim.x) {
      int pos = base + i;
      if (pos >= cap) pos -= cap;
      draws[i] = uint16_t(s.stream_mod[pos]);
    }
  }
  __syncthreads();
  const long long t2 = clock64();
  if (!parallel_done && tid < 32) {
    const int lane = tid;
    const uint32_t* __restrict__ smod = s.stream_mod;
    const uint64_t* __restrict__ ckey = s.c_key;
    long long gen_wp = wp;
    int best = s.best[0];
    uint64_t best_key = keys[best];
    int di = 0, b = 0;
    int failed = 0;
    int stage_begin = 0, stage_end = 0;
    auto stage = [&]() {  // child keys [b, b + 1024) into shared memory
      __syncwarp();
      stage_begin = b;
      stage_end = min(B, b + 1024);
      for (int i = lane; i < stage_end - stage_begin; i += 32) ck_stage[i] = ckey[stage_begin + i];
      __syncwarp();
    };
    while (b < B && !failed) {
      while (rs == 2 && b < B && di + 64 <= avail) {
        if (b + 32 > stage_end) stage();
        const int cnt = min(32, B - b);
        const bool live = lane < cnt;
        const int d0 = live ? int(draws[di + 2 * lane]) : -1 - 2 * lane;
        const int d1 = live ? int(draws[di + 2 * lane + 1]) : -2 - 2 * lane;
        const int latest = latest_overlap(d0, d1);
        const unsigned omask = __ballot_sync(kFull, live && latest >= 0);
        const int first_overlap = omask ? __ffs(omask) - 1 : cnt;
        const uint64_t ck = live ? ck_stage[b - stage_begin + lane] : ~0ULL;
        const int valid = place_segment(keys, placed, b, 0, first_overlap, max(d0, 0), max(d1, 0), ck, best,
                                        best_key);
        if (valid == 0) break;  // lane 0's victim is the best: the sequential loop redraws
        b += valid;
        di += 2 * valid;
      }
      if (b >= B) break;
      // sequential placement (lane 0): one child after a window stop, or every
      // remaining child past the staged draws / with another replacement size
      __syncwarp();
      if (lane == 0) {
        auto draw = [&](int idx) -> int {
          if (idx < avail) return draws[idx];
          const long long pos = rp + idx;
          while (pos >= gen_wp) {  // ran ahead of the buffer: one serial block
            mt_block_serial(s, mt, gen_wp);
            gen_wp += 312;
          }
          return int(smod[pos % cap]);
        };
        const bool rest = rs != 2 || di + 64 > avail;
        do {
          const uint64_t ck = ckey[b];
          int v = -1;
          for (int guard = 0; guard < (1 << 20); ++guard) {
            int worst = draw(di++);
            uint64_t kw = keys[worst];
            for (int i = 1; i < rs; ++i) {
              const int c = draw(di++);
              const uint64_t kc = keys[c];
              if (kw < kc || (kw == kc && worst < c)) { worst = c; kw = kc; }
            }
            if (worst != best) { v = worst; break; }
          }
          if (v < 0) { failed = 1; break; }
          keys[v] = ck;
          placed[v] = b;
          if (ck < best_key || (ck == best_key && v < best)) { best = v; best_key = ck; }
          ++b;
        } while (rest && b < B);
      }
      __syncwarp();
      b = __shfl_sync(kFull, b, 0);
      di = __shfl_sync(kFull, di, 0);
      best = __shfl_sync(kFull, best, 0);
      best_key = __shfl_sync(kFull, best_key, 0);
      gen_wp = __shfl_sync(kFull, gen_wp, 0);
      failed = __shfl_sync(kFull, failed, 0);
    }
    __syncwarp();
    if (lane == 0) {
      // the next round's variation seed: the raw output at the next position
      const long long pos = rp + di;
      while (pos >= gen_wp) {
        mt_block_serial(s, mt, gen_wp);
        gen_wp += 312;
      }
      s.round_seed[0] = s.stream[pos % cap];
      shared_best = best;
      shared_pos = pos + 1;
      shared_wp = gen_wp;
      shared_fail = failed;
    }
  }
  __syncthreads();
  const long long t3 = clock64();
  if (tid == 0) {
    if (shared_fail) raise_error(s, 40);
    s.best[0] = shared_best;
    stream_ptrs(s)[0] = shared_pos;
    stream_ptrs(s)[1] = shared_wp;
  }
  for (int i = tid; i < 312; i += blockDim.x) s.mt[i] = mt[i];
  if (tid == 0) {
    const int r = s.round[0] + 1;
    s.round[0] = r;
    if (r >= s.total_rounds) s.round[2] = 1;
    // SM clock cycles of the placement phases: generation, parallel
    // placement (and draw staging), windowed placement
    atomicAdd(reinterpret_cast<unsigned long long*>(&s.counters[4]), (unsigned long long)(t1 - t0));
    atomicAdd(reinterpret_cast<unsigned long long*>(&s.counters[5]), (unsigned long long)(t2 - t1));
    atomicAdd(reinterpret_cast<unsigned long long*>(&s.counters[6]), (unsigned long long)(t3 - t2));
  }
}

// after_cluster: the cluster placement ran first; return if it placed the
// round (place_state 1), replay it on the exact windowed path if it found a
// redraw (2), or place it here if it did not take it (0).
__global__ void __launch_bounds__(kPlaceThreads, 1) k_place(const SearchDesc* descs, int n, int dyn_bytes,
                                                            int after_cluster) {
  extern __shared__ __align__(16) uint64_t place_keys[];
  __shared__ PlaceShared sh;
  const SearchDesc& s = descs[blockIdx.x];
  if (!search_live(s)) return;
  const int state = after_cluster ? *s.place_state : 0;
  if (state == 1) return;
  if (s.B <= kPlaceThreads) place_round<1>(s, sh, place_keys, dyn_bytes, state == 2);
  else place_round<4>(s, sh, place_keys, dyn_bytes, state == 2);
}

// The children's two drawn members for this round, from the run generator's
// residues (draws 2j and 2j + 1 after the read position).
__device__ __forceinline__ uint32_t child_draws(const SearchDesc& s, int base, int j) {
  const int cap = s.stream_capacity;
  int p0 = base + 2 * j, p1 = p0 + 1;
  if (p0 >= cap) p0 -= cap;
  if (p1 >= cap) p1 -= cap;
  return s.stream_mod[p0] | (s.stream_mod[p1] << 16);
}

// Placement levels of a round, found before the children's keys exist.  A
// child can be placed once every earlier child that drew one of its members
// is placed: its level is one more than the largest level among those, which
// depends on the draws alone.  So this runs on the side stream, once the run
// generator has topped up the stream, while the children are still being
// varied and evaluated; k_place then only compares and writes keys, level by
// level.  Levels are found as the placement would find them: each level,
// every pending child claims both its members with a level-tagged atomicMin
// on the member's owner word, and a child that owns both is at this level.
// The owner words alternate between two arrays by level parity: a thread that
// has moved on to level L + 1 claims in the other array, so its claims never
// disturb a slower thread still checking level L (and the array of level L
// is claimed again only after barrier L + 1, which every check of level L
// precedes).  The levels are therefore the exact longest-path levels,
// whatever the timing.
// level_plan: [0] the round + 1 the levels belong to, [1] their number.
//
// In one block, for rounds of at most kLevelsSmall children whose two banks
// fit its shared memory.
__host__ __device__ __forceinline__ bool levels_small(const SearchDesc& s) { return s.B <= kLevelsSmall && s.P <= kLevelsSmall; }
__global__ void __launch_bounds__(kClusterThreads) k_place_levels_small(const SearchDesc* descs, int n) {
  __shared__ int32_t owner[2][kLevelsSmall];
  const SearchDesc& s = descs[blockIdx.x];
  if (!search_live(s) || !levels_small(s)) return;
  const int P = s.P, B = s.B, tid = threadIdx.x;
  const long long rp = stream_ptrs(s)[0], wp = stream_ptrs(s)[1];
  if (!levels_apply(s, rp, wp)) return;
  for (int m = tid; m < P; m += blockDim.x) owner[0][m] = owner[1][m] = 0x7fffffff;
  const int base = int(rp % s.stream_capacity);
  uint32_t cand[kClusterPer];
  uint32_t pending = 0;
#pragma unroll
  for (int t = 0; t < kClusterPer; ++t) {
    const int j = tid + t * kClusterThreads;
    cand[t] = 0;
    if (j < B) {
      cand[t] = child_draws(s, base, j);
      pending |= 1u << t;
    }
  }
  __syncthreads();
  int level = 0;
  for (; level <= B; ++level) {
    const int tag = (0x7fff - level) << 16;
    int32_t* const claims = owner[level & 1];
#pragma unroll
    for (int t = 0; t < kClusterPer; ++t)
      if (pending >> t & 1) {
        atomicMin(&claims[cand[t] & 0xffff], tag | (tid + t * kClusterThreads));
        atomicMin(&claims[cand[t] >> 16], tag | (tid + t * kClusterThreads));
      }
    if (!__syncthreads_or(pending != 0)) break;
#pragma unroll
    for (int t = 0; t < kClusterPer; ++t) {
      const int mine = tag | (tid + t * kClusterThreads);
      if ((pending >> t & 1) && claims[cand[t] & 0xffff] == mine && claims[cand[t] >> 16] == mine) {
        s.child_level[tid + t * kClusterThreads] = int16_t(level);
        pending &= ~(1u << t);
      }
    }
  }
  if (tid == 0) {
    s.level_plan[1] = level;  // levels 0 .. level - 1 hold every child
    s.level_plan[0] = s.round[0] + 1;
  }
}
// In a cluster of kPlaceCtas blocks that share their shared memory, for the
// others: member m's owner words live in block m % kPlaceCtas.
__global__ void __cluster_dims__(kPlaceCtas, 1, 1) __launch_bounds__(kClusterThreads, 1)
    k_place_levels(const SearchDesc* descs, int n) {
  extern __shared__ __align__(16) int32_t lv_owner[];
  __shared__ int ready_count[3];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = int(cluster.block_rank());
  const SearchDesc& s = descs[blockIdx.x / kPlaceCtas];
  if (!search_live(s)) return;  // the same for every block of the cluster
  const int P = s.P, B = s.B;
  const int tid = threadIdx.x, lane = tid & 31;
  const long long rp = stream_ptrs(s)[0], wp = stream_ptrs(s)[1];
  if (levels_small(s) || !levels_apply(s, rp, wp)) return;
  const int local_P = (P + kPlaceCtas - 1) / kPlaceCtas;
  for (int i = tid; i < 2 * local_P; i += blockDim.x) lv_owner[i] = 0x7fffffff;
  if (tid == 0) ready_count[0] = ready_count[1] = ready_count[2] = 0;
  const int begin = (rank * kClusterThreads + tid) * kClusterPer;
  const int base = int(rp % s.stream_capacity);
  uint32_t cand[kClusterPer];
  uint32_t pending = 0;
#pragma unroll
  for (int t = 0; t < kClusterPer; ++t) {
    cand[t] = 0;
    if (begin + t < B) {
      cand[t] = child_draws(s, base, begin + t);
      pending |= 1u << t;
    }
  }
  // owner word of member m for levels of parity `par`
  auto owner_at = [&](int m, int par) -> int* {
    return cluster.map_shared_rank(lv_owner, m % kPlaceCtas) + par * local_P + m / kPlaceCtas;
  };
  int* counter0 = cluster.map_shared_rank(ready_count, 0);
  int16_t* __restrict__ level_of = s.child_level;
  cluster.sync();
  // one cluster barrier per level; three count slots rotate: a level adds to
  // its own, reads the one before's and clears the next
  int left = B, level = 0;
  for (; level <= B; ++level) {
    const int tag = (0x7fff - level) << 16, par = level & 1;
#pragma unroll
    for (int t = 0; t < kClusterPer; ++t)
      if (pending >> t & 1) {
        atomicMin(owner_at(int(cand[t] & 0xffff), par), tag | (begin + t));
        atomicMin(owner_at(int(cand[t] >> 16), par), tag | (begin + t));
      }
    cluster.sync();
    if (level > 0) {
      left -= counter0[(level - 1) % 3];
      if (left == 0) break;
    }
    if (rank == 0 && tid == 0) ready_count[(level + 1) % 3] = 0;
    uint32_t ready = 0;
#pragma unroll
    for (int t = 0; t < kClusterPer; ++t)
      if ((pending >> t & 1) && *owner_at(int(cand[t] & 0xffff), par) == (tag | (begin + t)) &&
          *owner_at(int(cand[t] >> 16), par) == (tag | (begin + t))) {
        ready |= 1u << t;
        level_of[begin + t] = int16_t(level);
      }
    pending &= ~ready;
    int placed_here = __popc(ready);
    for (int o = 16; o; o >>= 1) placed_here += __shfl_xor_sync(kFull, placed_here, o);
    if (lane == 0 && placed_here) atomicAdd(counter0 + level % 3, placed_here);
  }
  if (rank == 0 && tid == 0) {
    s.level_plan[1] = level;  // levels 0 .. level - 1 hold every child
    s.level_plan[0] = s.round[0] + 1;
  }
  cluster.sync();  // no block leaves while another may still read its shared memory
}

// Cluster placement: the level-parallel placement of place_round, spread over
// a cluster of kPlaceCtas blocks that share their shared memory, for rounds
// of at least kClusterMinChildren children.  Member m's key lives in block
// m % kPlaceCtas; thread g of the cluster owns children [2g, 2g + 2), so the
// blocks hold the children in order.  Each level is a cluster barrier after
// the level's children have placed (remote key reads and writes).  The
// running best before each child is a scan inside each block plus a prefix
// over the blocks' totals.  When a child would have redrawn (place_state 2)
// k_place replays the round on the exact path; another replacement size or a
// stream short of draws is left to k_place (place_state 0).  On success this
// kernel finishes the round as k_place does (best member, stream position,
// next seed).
__global__ void __cluster_dims__(kPlaceCtas, 1, 1) __launch_bounds__(kClusterThreads, 1)
    k_place_cluster(const SearchDesc* descs, int n) {
  extern __shared__ __align__(16) uint64_t cl_keys[];
  __shared__ uint64_t scan_key[32];
  __shared__ int scan_idx[32];
  __shared__ uint64_t cta_key[kPlaceCtas];  // block totals (read from block 0)
  __shared__ int cta_idx[kPlaceCtas];
  __shared__ int redraw_at;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = int(cluster.block_rank());
  const SearchDesc& s = descs[blockIdx.x / kPlaceCtas];
  if (!search_live(s)) return;  // the same for every block of the cluster
  const long long t0 = clock64();
  const int P = s.P, B = s.B, cap = s.stream_capacity;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long long rp = stream_ptrs(s)[0], wp = stream_ptrs(s)[1];
  const int begin = (rank * kClusterThreads + tid) * kClusterPer;
  uint64_t kv[kClusterPer];  // the children's keys
#pragma unroll
  for (int t = 0; t < kClusterPer; ++t) kv[t] = begin + t < B ? s.c_key[begin + t] : ~0ULL;
  // the levels come from k_place_levels, run earlier in this round
  if (B < kClusterMinChildren || !levels_apply(s, rp, wp) || s.level_plan[0] != s.round[0] + 1) {
    if (rank == 0 && tid == 0) *s.place_state = 0;
    return;  // the same decision in every block
  }
  const int n_levels = s.level_plan[1];
  const int local_P = (P + kPlaceCtas - 1) / kPlaceCtas;
  uint64_t* keys = cl_keys;
  for (int i = tid; i < local_P; i += blockDim.x) {
    const int m = i * kPlaceCtas + rank;
    keys[i] = m < P ? s.key[m] : ~0ULL;
  }
  int32_t* __restrict__ placed = s.placed;
  for (int m = rank * kClusterThreads + tid; m < P; m += kPlaceCtas * kClusterThreads) placed[m] = -1;
  if (tid == 0) redraw_at = 0x7fffffff;
  const int base = int(rp % cap);
  uint32_t cand[kClusterPer];
  int lvl[kClusterPer];  // the children's placement levels
#pragma unroll
  for (int t = 0; t < kClusterPer; ++t) {
    const int j = begin + t;
    cand[t] = 0;
    lvl[t] = -1;
    if (j < B) {
      cand[t] = child_draws(s, base, j);
      lvl[t] = s.child_level[j];
    }
  }
  auto key_at = [&](int m) -> uint64_t* { return cluster.map_shared_rank(keys, m % kPlaceCtas) + m / kPlaceCtas; };
  cluster.sync();
  const long long level_start = clock64();
  // Level by level: the children of level L read both members' keys, the
  // worse member takes the child's key; a cluster barrier then makes the
  // writes visible to level L + 1.  Children of one level draw disjoint
  // members, so no two of them touch the same key.
  const int levels_run = n_levels;
  for (int level = 0; level < n_levels; ++level) {
#pragma unroll
    for (int t = 0; t < kClusterPer; ++t)
      if (lvl[t] == level) {
        const int d0 = int(cand[t] & 0xffff), d1 = int(cand[t] >> 16);
        const uint64_t k0 = *key_at(d0), k1 = *key_at(d1);
        // worst of the pair: the second replaces the first when the first is better
        const int v = (k0 < k1 || (k0 == k1 && d0 < d1)) ? d1 : d0;
        *key_at(v) = kv[t];
        placed[v] = begin + t;
        cand[t] = uint32_t(v);
      }
    cluster.sync();
  }
  const long long level_end = clock64();
  // best member before each child: (key, victim) minimum of this thread's
  // children, a warp scan, a block scan, then the blocks before this one
  uint64_t mk = ~0ULL;
  int mv = 0x7fffffff;
#pragma unroll
  for (int t = 0; t < kClusterPer; ++t)
    if (begin + t < B && key_before(kv[t], int(cand[t]), mk, mv)) { mk = kv[t]; mv = int(cand[t]); }
  for (int o = 1; o < 32; o <<= 1) {
    const uint64_t uk = __shfl_up_sync(kFull, mk, o);
    const int uv = __shfl_up_sync(kFull, mv, o);
    if (lane >= o && key_before(uk, uv, mk, mv)) { mk = uk; mv = uv; }
  }
  constexpr int kWarps = kClusterThreads / 32;
  if (lane == 31) { scan_key[warp] = mk; scan_idx[warp] = mv; }
  __syncthreads();
  if (warp == 0) {
    uint64_t wk = lane < kWarps ? scan_key[lane] : ~0ULL;
    int wv = lane < kWarps ? scan_idx[lane] : 0x7fffffff;
    for (int o = 1; o < 32; o <<= 1) {
      const uint64_t uk = __shfl_up_sync(kFull, wk, o);
      const int uv = __shfl_up_sync(kFull, wv, o);
      if (lane >= o && key_before(uk, uv, wk, wv)) { wk = uk; wv = uv; }
    }
    scan_key[lane] = wk;
    scan_idx[lane] = wv;
    if (lane == kWarps - 1) {
      *cluster.map_shared_rank(cta_key + rank, 0) = wk;
      *cluster.map_shared_rank(cta_idx + rank, 0) = wv;
    }
  }
  cluster.sync();
  const int best0 = s.best[0];
  const uint64_t best0_key = s.key[best0];
  int bv = best0;
  uint64_t bk = best0_key;
  {
    const uint64_t* tot_key = cluster.map_shared_rank(cta_key, 0);
    const int* tot_idx = cluster.map_shared_rank(cta_idx, 0);
    for (int r = 0; r < rank; ++r)
      if (key_before(tot_key[r], tot_idx[r], bk, bv)) { bk = tot_key[r]; bv = tot_idx[r]; }
    const uint64_t lk = __shfl_up_sync(kFull, mk, 1);
    const int lv = __shfl_up_sync(kFull, mv, 1);
    if (lane > 0 && key_before(lk, lv, bk, bv)) { bk = lk; bv = lv; }
    if (warp > 0 && key_before(scan_key[warp - 1], scan_idx[warp - 1], bk, bv)) {
      bk = scan_key[warp - 1];
      bv = scan_idx[warp - 1];
    }
  }
  // a child whose victim is the best member before it would have redrawn;
  // the earliest such child is noted in every block, so that no block reads
  // another's shared memory after the last cluster barrier
  bool hit = false;
#pragma unroll
  for (int t = 0; t < kClusterPer; ++t)
    if (!hit && begin + t < B) {
      const int v = int(cand[t]);
      if (v == bv) {
        for (int r = 0; r < kPlaceCtas; ++r) atomicMin(cluster.map_shared_rank(&redraw_at, r), begin + t);
        hit = true;
      } else if (key_before(kv[t], v, bk, bv)) {
        bk = kv[t];
        bv = v;
      }
    }
  cluster.sync();
  const bool done = redraw_at == 0x7fffffff;
  if (rank == 0 && tid == 0) {
    *s.place_state = done ? 1 : 2;
    if (done) {
      const uint64_t* tot_key = cta_key;
      int fv = best0;
      uint64_t fk = best0_key;
      for (int r = 0; r < kPlaceCtas; ++r)
        if (key_before(tot_key[r], cta_idx[r], fk, fv)) { fk = tot_key[r]; fv = cta_idx[r]; }
      s.best[0] = fv;
      // the next round's seed: the raw output after the 2B placement draws
      const long long pos = rp + 2LL * B;
      s.round_seed[0] = s.stream[pos % cap];
      stream_ptrs(s)[0] = pos + 1;
      const int r = s.round[0] + 1;
      s.round[0] = r;
      if (r >= s.total_rounds) s.round[2] = 1;
      atomicAdd(reinterpret_cast<unsigned long long*>(&s.counters[5]), (unsigned long long)(clock64() - t0));
      atomicAdd(reinterpret_cast<unsigned long long*>(&s.counters[14]), (unsigned long long)(level_end - level_start));
      atomicAdd(reinterpret_cast<unsigned long long*>(&s.counters[7]), (unsigned long long)levels_run);
    }
  }
}

// ------------------------------------------------------------ row evaluation
struct PackedRow {
  uint32_t node, constant;  // the row's first construction expression and constant
  int32_t len;              // its node and constant counts, as make_len packs them
};
static_assert(sizeof(PackedRow) == 12, "packed rows are uploaded as 12 bytes each");

// The packed rows of a row evaluation as node words, constants and lengths,
// a warp per row: evaluation reads the construction expression, the arity and
// the constant flag only.  Bound by the launch at a few rows and by the 16
// bytes written per node at many.
__global__ void k_unpack_rows(const SearchDesc* desc, const int64_t* __restrict__ constants,
                              const PackedRow* __restrict__ rows, const uint16_t* __restrict__ origins) {
  const int r = int((size_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  const SearchDesc& s = *desc;
  if (r >= s.P) return;
  const PackedRow row = rows[r];
  const int n = len_nodes(row.len), nc = len_consts(row.len);
  const gagp_expression* __restrict__ ex = s.ex;
  for (int i = lane; i < n; i += 32) {
    const int o = origins[row.node + i];
    s.node[size_t(r) * s.stride + i] = uint64_t(uint32_t(o)) | (uint64_t(uint32_t(ex[o].arity) & 0xfu) << 48) |
                                       (uint64_t(ex[o].kind == EK_CONSTANT) << 52) | (uint64_t(kNoClass) << 53);
  }
  for (int k = lane; k < nc; k += 32) s.cval[size_t(r) * s.stride + k] = constants[row.constant + k];
  if (lane == 0) s.len[r] = row.len;
}

// ------------------------------------------------------------ result export
// The final population ranked as the reference ranks it (by ranking key,
// ties by member index, selection.cpp:10-20): a member's rank is the number
// of members before it, counted against shared-memory tiles of the keys.
constexpr int kRankTile = 1024;
__global__ void __launch_bounds__(128) k_rank_members(const SearchDesc* desc, int32_t* rank) {
  __shared__ uint64_t tile[kRankTile];
  const SearchDesc& s = *desc;
  const int P = s.P;
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t mk = m < P ? s.key[m] : 0;
  int r = 0;
  for (int base = 0; base < P; base += kRankTile) {
    __syncthreads();
    for (int i = threadIdx.x; i < kRankTile; i += blockDim.x) tile[i] = base + i < P ? s.key[base + i] : ~0ULL;
    __syncthreads();
    const int lim = min(kRankTile, P - base);
    if (m < P)
      for (int j = 0; j < lim; ++j) {
        const uint64_t k = tile[j];
        r += k < mk || (k == mk && base + j < m);
      }
  }
  if (m < P) rank[m] = r;
}

// Each member's statistics and transport row (construction expressions and
// constants, `width` entries per row, zero past its counts) at its rank:
// a warp per member.
__global__ void k_export_members(const SearchDesc* desc, const int32_t* rank, int width, double* fitness,
                                 int32_t* wrong, int32_t* nodes, int32_t* node_counts, int32_t* constant_counts,
                                 int32_t* origins, int64_t* constants) {
  const int m = int((size_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  const SearchDesc& s = *desc;
  if (m >= s.P) return;
  const int r = rank[m];
  const int32_t l = s.len[m];
  const int n = len_nodes(l), nc = len_consts(l);
  if (lane == 0) {
    fitness[r] = s.fitness[m];
    wrong[r] = s.has_wrong ? int32_t(s.wrong[m]) : -1;
    nodes[r] = s.fixed_nodes + n;
    node_counts[r] = n;
    constant_counts[r] = nc;
  }
  const uint64_t* node = s.node + size_t(m) * s.stride;
  const int64_t* cval = s.cval + size_t(m) * s.stride;
  for (int i = lane; i < width; i += 32) {
    origins[size_t(r) * width + i] = i < n && i < s.stride ? int32_t(node[i] & 0xffffu) : 0;
    constants[size_t(r) * width + i] = i < nc && i < s.stride ? cval[i] : 0;
  }
}

// commit_batch (phase_population_cpu.cpp:382-394): placed child rows replace
// members.  Thread per member.
constexpr int kCommitLanes = 16;  // threads per member row
__global__ void k_commit(const SearchDesc* descs, const int32_t* off, int n) {
  const size_t gid = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const int item = int(gid / kCommitLanes), lane = int(gid % kCommitLanes);
  if (item >= off[n]) return;
  const int si = find_search(off, n, item);
  const SearchDesc& s = descs[si];
  if (s.round[3]) return;
  const int m = item - off[si];
  // this round's member index is spent: its slots start the next round empty
  if (s.mtab) {
    const int e = m * kCommitLanes + lane;
    if (e <= s.mtab_mask) s.mtab[e] = 0;
  }
  const int b = s.placed[m];
  if (b < 0) return;
  // the row's threads copy consecutive slots: coalesced reads and writes
  const int32_t l = s.clen[b];
  const uint64_t* from = s.cnode + size_t(b) * s.stride;
  const int64_t* cfrom = s.ccval + size_t(b) * s.stride;
  uint64_t* to = s.node + size_t(m) * s.stride;
  int64_t* cto = s.cval + size_t(m) * s.stride;
  for (int i = lane; i < len_nodes(l); i += kCommitLanes) to[i] = from[i];
  for (int i = lane; i < len_consts(l); i += kCommitLanes) cto[i] = cfrom[i];
  if (lane == 0) {
    s.len[m] = l;
    if (!s.generational) {  // k_gen_place has copied these
      s.fitness[m] = s.c_fitness[b];
      s.wrong[m] = s.c_wrong[b];
      s.nodes[m] = s.c_nodes[b];
      s.key[m] = s.c_key[b];
    }
  }
}

// ----------------------------------------------------------- generational
// The generational schedule's placement (reproduce, phase_population_cpu.cpp:
// 269-312, then the next evaluate's reuse, :243-265): child i becomes member
// i with its result.  Runs after the lowering, which read the members'
// results for the reused children; k_commit then copies the rows.
__global__ void k_gen_place(const SearchDesc* descs, const int32_t* off, int n) {
  const int item = blockIdx.x * blockDim.x + threadIdx.x;
  if (item >= off[n]) return;
  const int si = find_search(off, n, item);
  const SearchDesc& s = descs[si];
  if (!search_live(s)) return;
  const int m = item - off[si];
  s.fitness[m] = s.c_fitness[m];
  s.wrong[m] = s.c_wrong[m];
  s.nodes[m] = s.c_nodes[m];
  s.key[m] = s.c_key[m];
  s.placed[m] = m;
}

// End of a generational round, one block per search: the next round's
// elites and best member, its variation seed (the next run-generator output,
// one per generation as run_phase_population draws rng() per reproduce,
// evolve.cpp:300-301) and the round count.
__global__ void k_gen_finish(const SearchDesc* descs, int n) {
  __shared__ uint64_t mt[312], nw[312];
  __shared__ int32_t best_one[1];
  const SearchDesc& s = descs[blockIdx.x];
  if (!search_live(s)) return;
  if (s.elite_count > 0) {
    block_best_members(s, s.elite_count, s.elites);
  } else {
    block_best_members(s, 1, best_one);
  }
  __syncthreads();
  long long* head = stream_ptrs(s);
  const long long rp = head[0], wp = head[1];
  if (rp >= wp) {  // the run generator's next block (every 312 generations)
    for (int i = threadIdx.x; i < 312; i += blockDim.x) mt[i] = s.mt[i];
    __syncthreads();
    mt_block(s, mt, nw, wp);
    for (int i = threadIdx.x; i < 312; i += blockDim.x) s.mt[i] = mt[i];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    s.best[0] = s.elite_count > 0 ? s.elites[0] : best_one[0];
    s.round_seed[0] = s.stream[rp % s.stream_capacity];
    head[0] = rp + 1;
    if (rp >= wp) head[1] = wp + 312;
    const int done = s.round[0] + 1;
    s.round[0] = done;
    if (done >= s.total_rounds) s.round[2] = 1;
  }
}

}  // namespace gb
