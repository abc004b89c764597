// The CUDA side of the synthesis-database fill (sm_100a).
//
// Specs are processed stage by stage (plan.hpp). A team of blocks solves a whole stage on the device,
// with barriers between its phases and nothing for the host to decide.
// A limits grid of a Spec = per memory the lattice codes at which its result can change; a cell
// = one combination of slots; evaluating a candidate record at a cell = feasibility under the
// cell's limits, gather of the child rows at the children's limits, combine into a Cost,
// lexicographic minimum.
//   0. corners: below its corner a Spec has no implementation at all; every grid of the stage is
//      clipped there (phase_minsat, phase_records, phase_place_early);
//   1. once per stage, the records whose children all lie in earlier stages are solved on a grid
//      of their own - their thresholds plus the (shifted) breakpoints of those children's
//      finished tables - in no particular order: a warp takes a piece of one Spec's grid, stages
//      the Spec's records and the headers of their children in shared memory, orders the records by
//      a lower bound on their cost there, and its lanes take 32 cells at a time and walk the staged
//      records together as far as one can still gain (phase_early; phase_early_fused for small
//      teams); the real breakpoints of the result are found at once (phase_real_masks);
//   2. the rest - relayout Moves, whose body is a Spec of the same stage at strictly lower limits
//      - is solved on working grids: the real breakpoints of step 1's result, the thresholds of
//      those records and the shifted breakpoints of their children (phase_place_late), in sweeps
//      until one changes nothing (phase_sweep): the dependencies between cells form no cycle, so
//      that fixpoint is the direct solve;
//   3. breakpoints at which some pair of neighbouring cells differs are real
//      (phase_real_masks); 2-3 repeat for the Specs whose working grid still lacks a breakpoint
//      that a same-stage child turned out to have (phase_check_grids, phase_refine);
//   4. the grids are compacted to the real breakpoints and appended to the table (phase_count,
//      phase_compact).
// Step 3's fixpoint is exact: when every Spec's grid contains all thresholds and all shifted
// breakpoints of the computed tables of its children, induction over the limits lattice shows
// every computed cell equals the direct solve at every limit inside it.
//
// What the combine replaces in the reference (paths inside the Morello repository):
//   morello/src/scheduling/mod.rs:286-368     ActionSolver::compute_cost
//   morello/src/imp/loops.rs:207-242          loop main cost (serial, no boundary regions)
//   morello/src/memorylimits.rs:159-224,409-470  peak propagation, limit subtraction
//   morello/src/scheduling/select.rs:34-47    kernel-allocation feasibility
//   morello/src/search/reducer.rs:40-99       argmin on (Cost, ActionNum)
//   morello/src/db/pagecontents.rs:103-123    child lookup (here: an index computation)
//   precompute/src/main.rs:304-385            the stage loop (here: on the device)
// Integer-only work; no tensor cores.
#include "device_types.h"
#include "fill.hpp"
#include "devplan.hpp"
#include "host_threads.hpp"
#include "../../include/morello_b200.h"
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <algorithm>
#include <chrono>
#include <mutex>
#include <thread>
#include <type_traits>

namespace cg = cooperative_groups;

static_assert(MRL_STATIC_SCRATCH_BYTES == MRL_NOALLOC_MAX_BYTES,
              "the fixed device array and the limit the header promises are one number");

namespace {

constexpr int kBlock = 128;         // threads per block of the small kernels here
constexpr int kStageBlock = 1024;   // ... of the stage kernel: one block per SM (64 registers), so few arrive at a barrier
constexpr int kMaxPasses = 128;
constexpr int kMaxSweeps = 256;   // per pass; a dependency chain is shorter than the 70 diagonals of the limits lattice

__device__ __forceinline__ uint32_t sat_add(uint32_t a, uint32_t b) {
  uint32_t s = a + b;
  return s < a ? 0xFFFFFFFFu : s;
}
__device__ __forceinline__ uint32_t sat_mul(uint32_t a, uint32_t b) {
  unsigned long long p = (unsigned long long)a * b;
  return p > 0xFFFFFFFFull ? 0xFFFFFFFFu : (uint32_t)p;
}
// cpack: limit codes packed one per byte, RF in byte 0 .. GL in byte 3.
__device__ __forceinline__ uint32_t code_of(uint32_t cpack, uint32_t level) { return (cpack >> (8 * level)) & 0xFFu; }
// peaks word: RF in byte 3 .. GL in byte 0 (so that a plain u32 compare is lexicographic).
__device__ __forceinline__ uint32_t peak_shift(uint32_t level) { return 8 * (3 - level); }

// Code of the power-of-two-rounded line count x (0 -> 0, 1 -> 1, 2 -> 2, 3..4 -> 3, ...).
__device__ __forceinline__ uint32_t cache_code_ceil(uint32_t x) {
  if (x == 0) return 0;
  if (x == 1) return 1;
  return (32 - __clz(x - 1)) + 1;
}
__device__ __forceinline__ uint32_t cache_value(uint32_t code) { return code ? (1u << (code - 1)) : 0u; }

// The limit code a Move's children see in the memory it allocates in, given the parent's code
// there (at or above the Move's threshold): registers subtract, caches subtract and snap down
// to a power of two (morello/src/memorylimits.rs:409-436).
__device__ __forceinline__ uint32_t child_code(uint32_t level, uint32_t lv, uint32_t units) {
  return level < 2 ? lv - units : 32 - __clz(cache_value(lv) - units);
}

// Position of the n-th (0-based) set bit of m; m has more than n bits set.
__device__ __forceinline__ uint32_t nth_set_bit(uint32_t m, uint32_t n) {
  uint32_t pos = 0;
#pragma unroll
  for (int w = 16; w > 0; w >>= 1) {
    const uint32_t low = __popc(m & ((1u << w) - 1u));
    const bool up = n >= low;
    n -= up ? low : 0u;
    m = up ? (m >> w) : m;
    pos += up ? (uint32_t)w : 0u;
  }
  return pos;
}

__device__ __forceinline__ uint32_t sel4(uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t k) {
  return k == 0 ? a0 : (k == 1 ? a1 : (k == 2 ? a2 : a3));
}
__device__ __forceinline__ uint32_t below(uint32_t code) { return (2u << code) - 1u; }   // codes <= code

// Slot indices come out of cell numbers by division by slot counts (1 to 31). x / n = the high word of x *
// ceil(2^32 / n) while x * n < 2^32 (cells of a Spec < 2^20), three instructions instead of twenty.
__constant__ uint32_t kReciprocal[32] = {
#define MRL_R(n) (n) < 2 ? 0u : 0xFFFFFFFFu / ((n) < 2 ? 2u : (n)) + 1u
    MRL_R(0), MRL_R(1), MRL_R(2), MRL_R(3), MRL_R(4), MRL_R(5), MRL_R(6), MRL_R(7), MRL_R(8), MRL_R(9), MRL_R(10),
    MRL_R(11), MRL_R(12), MRL_R(13), MRL_R(14), MRL_R(15), MRL_R(16), MRL_R(17), MRL_R(18), MRL_R(19), MRL_R(20), MRL_R(21),
    MRL_R(22), MRL_R(23), MRL_R(24), MRL_R(25), MRL_R(26), MRL_R(27), MRL_R(28), MRL_R(29), MRL_R(30), MRL_R(31)
#undef MRL_R
};
// x / n, and x becomes x % n.
__device__ __forceinline__ uint32_t div_slots(uint32_t& x, uint32_t n) {
  const uint32_t q = n == 1 ? x : __umulhi(x, kReciprocal[n]);
  x -= q * n;
  return q;
}
// Slots of a cell (RF fastest) in a grid of n0 * n1 * n2 * .. slots.
__device__ __forceinline__ void cell_slots(uint32_t cell, uint32_t n0, uint32_t n1, uint32_t n2, uint32_t& s0, uint32_t& s1, uint32_t& s2, uint32_t& s3) {
  s0 = cell;
  s1 = div_slots(s0, n0);
  s2 = div_slots(s1, n1);
  s3 = div_slots(s2, n2);
}

// The running optimum of a cell: the row's three key words.
struct Best {
  uint32_t main, peaks, tail;
};
__device__ __forceinline__ bool key_less(uint32_t m, uint32_t p, uint32_t t, const Best& b) {
  if (m != b.main) return m < b.main;
  if (p != b.peaks) return p < b.peaks;
  return t < b.tail;
}

struct Tally {   // what a thread's solves touched
  uint32_t cands, lookups;
};

// Row `base` of the table: bit 63 set = a working row of the stage being solved.
#define MRL_TEMP_FLAG (1ull << 63)
__device__ __forceinline__ const MrlRow* row_at(const MrlRow* rows, const MrlRow* temp, unsigned long long base) {
  return ((base & MRL_TEMP_FLAG) ? temp : rows) + (base & ~MRL_TEMP_FLAG);
}

// Row of a child Spec at given limits: the cell whose breakpoints are the largest ones not
// above the limits. b_k = mask of the codes <= the limit's code in memory k. One 32-byte
// header and one 16-byte row. Plain loads: headers and working rows of the stage being solved
// are written by earlier phases of the same launch.
__device__ __forceinline__ const MrlRow* row_of(const MrlRow* rows, const MrlRow* temp, const uint4 m,
                                                unsigned long long base, uint32_t b0, uint32_t b1, uint32_t b2,
                                                uint32_t b3) {
  const uint32_t i0 = __popc(m.x & b0) - 1;
  const uint32_t i1 = __popc(m.y & b1) - 1;
  const uint32_t i2 = __popc(m.z & b2) - 1;
  const uint32_t i3 = __popc(m.w & b3) - 1;
  const uint32_t off = ((i3 * __popc(m.z) + i2) * __popc(m.y) + i1) * __popc(m.x) + i0;  // cells per Spec < 2^32
  return row_at(rows, temp, base) + off;
}
__device__ __forceinline__ uint4 lookup(const SpecHdr* hdrs, const MrlRow* rows, const MrlRow* temp, uint32_t child,
                                        uint32_t b0, uint32_t b1, uint32_t b2, uint32_t b3) {
  const uint4 m = *reinterpret_cast<const uint4*>(&hdrs[child]);
  const unsigned long long base = hdrs[child].row_base;
  return *reinterpret_cast<const uint4*>(row_of(rows, temp, m, base, b0, b1, b2, b3));
}

// One candidate record of a Spec at one limits point, for the verifier (the fill's is eval_staged):
// feasibility under the limits, the child rows at the children's limits, the combined Cost, and the
// running minimum. The headers of all children are requested together, then all rows: two round trips
// per candidate whatever the number of children.
__device__ __forceinline__ void eval_candidate(const SpecHdr* hdrs, const CandRec* __restrict__ cands, const MrlRow* rows,
                                               const MrlRow* temp, uint32_t rec, const uint4 a, uint32_t cpack,
                                               uint32_t bm0, uint32_t bm1, uint32_t bm2, uint32_t bm3, Best& best,
                                               Tally& tally) {
  const uint32_t action = a.x & 0xFFFFu, kind = (a.x >> 16) & 0xFFu, nchild = a.x >> 24;
  const uint32_t imm = a.y;
  const uint32_t level = a.z & 0xFFu, thr = (a.z >> 8) & 0xFFu, pcode = (a.z >> 16) & 0xFFu;
  const uint32_t units = a.w;
  const uint32_t lv = code_of(cpack, level);  // the cell's limit in `level`
  tally.cands++;
  uint32_t k_main, k_peaks, k_tail;
  if (kind == MRL_CK_LEAF) {
    if (lv < thr) return;
    k_main = imm;
    k_peaks = pcode << peak_shift(level);
    k_tail = (1u << 16) | action;
  } else {
    uint32_t c0 = bm0, c1 = bm1, c2 = bm2, c3 = bm3;
    const uint32_t sh = peak_shift(level);
    if (kind == MRL_CK_MOVE) {
      if (lv < thr) return;
      // Branch and bound: a Move costs at least its own base cost.
      if (imm > best.main) return;
      const uint32_t cb = below(child_code(level, lv, units));
      c0 = (level == 0) ? cb : c0;
      c1 = (level == 1) ? cb : c1;
      c2 = (level == 2) ? cb : c2;
      c3 = (level == 3) ? cb : c3;
    }
    const uint4 b = __ldg(reinterpret_cast<const uint4*>(&cands[rec]) + 1);
    const uint32_t ch1 = nchild > 1 ? b.y : b.x, ch2 = nchild > 2 ? b.z : b.x;   // absent children repeat the first
    const uint4 m0 = *reinterpret_cast<const uint4*>(&hdrs[b.x]);
    const uint4 m1 = *reinterpret_cast<const uint4*>(&hdrs[ch1]);
    const uint4 m2 = *reinterpret_cast<const uint4*>(&hdrs[ch2]);
    const unsigned long long base0 = hdrs[b.x].row_base, base1 = hdrs[ch1].row_base, base2 = hdrs[ch2].row_base;
    const uint4 r0 = *reinterpret_cast<const uint4*>(row_of(rows, temp, m0, base0, c0, c1, c2, c3));
    const uint4 r1 = *reinterpret_cast<const uint4*>(row_of(rows, temp, m1, base1, c0, c1, c2, c3));
    const uint4 r2 = *reinterpret_cast<const uint4*>(row_of(rows, temp, m2, base2, c0, c1, c2, c3));
    tally.lookups += nchild;
    if (r0.z == MRL_UNSAT || r1.z == MRL_UNSAT || r2.z == MRL_UNSAT) return;
    uint32_t depth;
    if (kind == MRL_CK_LOOP) {
      k_main = sat_mul(r0.x, imm);
      k_peaks = r0.y;
      depth = 1u;  // a single-body tile loop has depth 1 whatever its body's depth
    } else {
      k_main = (kind == MRL_CK_MOVE) ? sat_add(imm, r0.x) : r0.x;
      if (nchild > 1) k_main = sat_add(k_main, r1.x);
      if (nchild > 2) k_main = sat_add(k_main, r2.x);
      if (k_main > best.main) return;
      k_peaks = __vmaxu4(__vmaxu4(r0.y, r1.y), r2.y);
      if (kind == MRL_CK_MOVE) {
        // own allocation sits on top of the deepest child's peak in `level`; rounding to the
        // lattice is monotone, so max-then-round equals the reference's round-per-child
        const uint32_t cc = (k_peaks >> sh) & 0xFFu;
        const uint32_t ncode = level < 2 ? units + cc : cache_code_ceil(units + cache_value(cc));
        k_peaks = (k_peaks & ~(0xFFu << sh)) | (ncode << sh);
      }
      depth = min(max(max(r0.z >> 16, r1.z >> 16), r2.z >> 16) + 1u, 255u);
    }
    k_tail = (depth << 16) | action;
  }
  if (key_less(k_main, k_peaks, k_tail, best)) {
    best.main = k_main;
    best.peaks = k_peaks;
    best.tail = k_tail;
  }
}

// The direct solve of one (Spec, limits) point from the tables of the Spec's children: every
// candidate record of the Spec. cpack = the limits as lattice codes.
__device__ __forceinline__ Best solve_point(const SpecHdr* hdrs, const CandRec* __restrict__ cands, const MrlRow* rows,
                                            const MrlRow* temp, uint32_t spec, uint32_t cpack, Tally& tally) {
  const uint32_t bm0 = below(code_of(cpack, 0)), bm1 = below(code_of(cpack, 1)), bm2 = below(code_of(cpack, 2)),
                 bm3 = below(code_of(cpack, 3));
  const uint2 cl = *reinterpret_cast<const uint2*>(&hdrs[spec].cand_off);
  Best best = {MRL_UNSAT, MRL_UNSAT, MRL_UNSAT};
  for (uint32_t ci = 0; ci < cl.y; ci++) {
    const uint4 a = __ldg(reinterpret_cast<const uint4*>(&cands[cl.x + ci]));
    eval_candidate(hdrs, cands, rows, temp, cl.x + ci, a, cpack, bm0, bm1, bm2, bm3, best, tally);
  }
  return best;
}

// ---- working grids ---------------------------------------------------------------------

__device__ __forceinline__ void or_level(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3, uint32_t level,
                                         uint32_t bits) {
  r0 |= (level == 0) ? bits : 0u;
  r1 |= (level == 1) ? bits : 0u;
  r2 |= (level == 2) ? bits : 0u;
  r3 |= (level == 3) ? bits : 0u;
}

// Where a child's breakpoints in the destination memory of a Move show up in the parent: the
// child sees limit - units (registers) or that snapped down to a power of two (caches), so a
// child breakpoint at code b becomes the smallest parent code whose child code reaches b.
__device__ __forceinline__ uint32_t shift_mask(uint32_t cm, uint32_t level, uint32_t units, uint32_t top) {
  const uint32_t keep = (2u << top) - 1u;   // top <= 30
  if (level < 2) return units >= 32 ? 0u : (uint32_t)(((unsigned long long)cm << units) & keep);
  uint32_t out = 0;
#pragma unroll 1
  while (cm) {
    const uint32_t b = __ffs(cm) - 1;
    cm &= cm - 1;
    const unsigned long long v = (unsigned long long)cache_value(b) + units;
    if (v > 0x40000000ull) continue;
    const uint32_t code = cache_code_ceil((uint32_t)v);
    if (code <= top) out |= 1u << code;
  }
  return out;
}

// A run of stages, as one launch sees it; passed by value. The stage's counters (StageCtl) lie in the
// control block, or in shared memory when the team is one block.
struct StageArgs {
  SpecHdr* hdrs;
  const CandRec* cands;
  uint4* rmask;
  const uint8_t* mine;    // null: every Spec is computed here
  WorkItem* items;
  MrlRow* rows;
  MrlRow* temp;           // working rows; temp_cap rows further on, the grids of the unordered phase
  uint32_t* minsat;       // by Spec id: lower corner of the satisfiable region (see phase_minsat)
  StageSpec* sspec;       // by position in the stage
  uint4* changed[3];      // by position in the stage, three sweeps in turn: codes of the slots a sweep changed
  unsigned long long* block_sums;
  FillCtl* ctl;
  const uint2* stages;    // [first, end) Spec id of every stage
  uint32_t stage_lo, stage_hi;   // the stages of this launch
  uint32_t top_pack;
  uint32_t team;          // TEAM_*: what a barrier spans
  unsigned long long temp_cap, item_cap, row_cap;
  int solve, place;       // which halves to run
};
enum { TEAM_BLOCK = 0, TEAM_CLUSTER = 1, TEAM_GRID = 2 };

__device__ __forceinline__ bool computed_here(const StageArgs& a, uint32_t i) { return !a.mine || a.mine[i]; }

// Lower corner of a Spec's satisfiable region: per memory the smallest limit code at which any
// implementation exists at all, one byte each (RF in the low byte); 31 = none anywhere. More memory
// never loses an implementation, so every limits point with a coordinate below the corner is
// unsatisfiable. For a finished Spec the corner is exact (read off its table); for a Spec of the
// stage being solved it is a lower bound worked out from its candidates before anything is solved.
#define MRL_NEVER 31u
#define MRL_NEVER4 0x1F1F1F1Fu
__device__ __forceinline__ uint32_t corner_of(uint32_t pack, uint32_t k) { return (pack >> (8 * k)) & 0xFFu; }
// A cell with a limit below its Spec's corner has no implementation; no record needs to be read.
__device__ __forceinline__ bool below_corner(uint32_t corner, uint32_t cpack) { return __vcmpltu4(cpack, corner) != 0; }

// Exact corner of a Spec from its finished rows, by a warp. Along memory k the cell with the top slot
// in every other memory is satisfiable as soon as any cell with that slot in k is.
__device__ __forceinline__ uint32_t corner_from_rows(const uint4 m, const MrlRow* grid, uint32_t lane) {
  const uint32_t mm[4] = {m.x, m.y, m.z, m.w};
  uint32_t nn[4], st[4];
#pragma unroll
  for (int k = 0; k < 4; k++) nn[k] = __popc(mm[k]);
  st[0] = 1; st[1] = nn[0]; st[2] = nn[0] * nn[1]; st[3] = nn[0] * nn[1] * nn[2];
  uint32_t top = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) top += (nn[k] - 1) * st[k];
  uint32_t tail[4];
#pragma unroll
  for (int k = 0; k < 4; k++) tail[k] = lane < nn[k] ? grid[top - (nn[k] - 1 - lane) * st[k]].tail : MRL_UNSAT;   // at most 31 slots
  uint32_t pack = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const uint32_t sat = __ballot_sync(0xFFFFFFFFu, tail[k] != MRL_UNSAT);
    pack |= (sat ? nth_set_bit(mm[k], __ffs(sat) - 1) : MRL_NEVER) << (8 * k);
  }
  return pack;
}

// Corners of the Specs of an earlier stage whose rows came from several ranks.
__device__ __noinline__ void phase_minsat(const StageArgs& a, uint32_t lo, uint32_t hi, uint32_t gwarp, uint32_t gwarps) {
  const uint32_t lane = threadIdx.x & 31;
  #pragma unroll 1
  for (uint32_t i = lo + gwarp; i < hi; i += gwarps) {
    const uint32_t corner = corner_from_rows(*reinterpret_cast<const uint4*>(&a.hdrs[i]), a.rows + a.hdrs[i].row_base, lane);
    if (lane == 0) a.minsat[i] = corner;
  }
}

// What one record needs at least, per memory: its threshold; its children's corners, shifted by what
// a Move takes. NEVER4: no limits inside the lattice satisfy it. Same-stage children: corner zero
// (bounds = false), or what the round before worked out for them.
__device__ __forceinline__ uint32_t record_corner(const StageArgs& a, uint32_t lo, const uint4 c, const uint4 b, bool bounds) {
  const uint32_t kind = (c.x >> 16) & 0xFFu, nchild = c.x >> 24;
  const uint32_t level = c.z & 0xFFu, thr = (c.z >> 8) & 0xFFu, units = c.w;
  uint32_t q = (kind == MRL_CK_LEAF || kind == MRL_CK_MOVE) ? thr << (8 * level) : 0u;
#pragma unroll 1
  for (uint32_t j = 0; j < nchild; j++) {
    const uint32_t child = j == 0 ? b.x : (j == 1 ? b.y : b.z);
    uint32_t e = (child < lo || bounds) ? a.minsat[child] : 0u;
    if ((e & 0xFFu) == MRL_NEVER) return MRL_NEVER4;
    if (kind == MRL_CK_MOVE) {
      const uint32_t el = corner_of(e, level);
      // the smallest code whose child code reaches el
      const uint32_t sh = el == 0 ? 0u : (level < 2 ? el + units : cache_code_ceil(cache_value(el) + units));
      if (sh > code_of(a.top_pack, level)) return MRL_NEVER4;
      e = (e & ~(0xFFu << (8 * level))) | (sh << (8 * level));
    }
    q = __vmaxu4(q, e);
  }
  return q;
}
__device__ __forceinline__ uint32_t warp_min4(uint32_t v) {
  for (int o = 16; o > 0; o >>= 1) v = __vminu4(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
  return v;
}

// Clips a grid at the corner: below it everything is unsatisfiable, so one cell [0, corner) per
// memory is enough.
__device__ __forceinline__ uint4 clip_at_corner(uint4 nm, uint32_t corner) {
  const uint32_t k0 = corner_of(corner, 0), k1 = corner_of(corner, 1), k2 = corner_of(corner, 2), k3 = corner_of(corner, 3);
  if (k0 == MRL_NEVER) return make_uint4(1u, 1u, 1u, 1u);   // unsatisfiable at every limit: a single cell
  if (k0) nm.x = (nm.x & ~((1u << k0) - 1u)) | 1u | (1u << k0);
  if (k1) nm.y = (nm.y & ~((1u << k1) - 1u)) | 1u | (1u << k1);
  if (k2) nm.z = (nm.z & ~((1u << k2) - 1u)) | 1u | (1u << k2);
  if (k3) nm.w = (nm.w & ~((1u << k3) - 1u)) | 1u | (1u << k3);
  return nm;
}

// ORs into r the breakpoints one record puts into its Spec's grid: its own threshold, and its
// children's breakpoints (for a Move, shifted in the memory it allocates in). Children of
// finished stages contribute their final masks, same-stage children what rmask holds for them.
__device__ __forceinline__ void record_breakpoints(const StageArgs& a, uint32_t lo, const uint4 c, const uint4 b, uint4& r) {
  const uint32_t kind = (c.x >> 16) & 0xFFu, nchild = c.x >> 24;
  const uint32_t level = c.z & 0xFFu, thr = (c.z >> 8) & 0xFFu, units = c.w;
  if (kind == MRL_CK_LEAF || kind == MRL_CK_MOVE) or_level(r.x, r.y, r.z, r.w, level, 1u << thr);
#pragma unroll 1
  for (uint32_t j = 0; j < nchild; j++) {
    const uint32_t child = j == 0 ? b.x : (j == 1 ? b.y : b.z);
    const uint4 cm = child < lo ? *reinterpret_cast<const uint4*>(&a.hdrs[child]) : a.rmask[child];
    if (kind == MRL_CK_MOVE) {
      const uint32_t s = shift_mask(sel4(cm.x, cm.y, cm.z, cm.w, level), level, units, code_of(a.top_pack, level));
      r.x |= (level == 0) ? s : cm.x;
      r.y |= (level == 1) ? s : cm.y;
      r.z |= (level == 2) ? s : cm.z;
      r.w |= (level == 3) ? s : cm.w;
    } else {
      r.x |= cm.x; r.y |= cm.y; r.z |= cm.z; r.w |= cm.w;
    }
  }
}
__device__ __forceinline__ uint4 warp_or(uint4 r) {
  r.x = __reduce_or_sync(0xFFFFFFFFu, r.x);
  r.y = __reduce_or_sync(0xFFFFFFFFu, r.y);
  r.z = __reduce_or_sync(0xFFFFFFFFu, r.z);
  r.w = __reduce_or_sync(0xFFFFFFFFu, r.w);
  return r;
}
__device__ __forceinline__ unsigned long long cells_of(const uint4 m) {
  return (unsigned long long)__popc(m.x) * __popc(m.y) * __popc(m.z) * __popc(m.w);
}

// A candidate record whose body is a Spec of the same stage (a relayout Move): the planner flags
// it and stores these records after all others, dearest first.
__device__ __forceinline__ bool is_late(const uint4 a) { return (a.z >> 24) & 1u; }

// The Specs a warp of a per-Spec phase takes at a time: as many as keep all warps busy, at most one
// per lane.
__device__ __forceinline__ uint32_t group_size(uint32_t n, uint32_t gwarps) { return max(1u, min(32u, (n + gwarps - 1) / gwarps)); }
// Cells per work item of a grid, as a power of two times 32 (0 to 5: 32 to MRL_ITEM_CELLS cells). An item's
// records are staged and bounded once, so items are long while there are enough of them: some four for
// every warp if the stage's other grids are as large as this one, and 128 cells a grid, the average, are
// taken where it is smaller or has more same-stage records than a batch (then its cells cost several
// times those of others, and long items leave warps idle at the barrier). 8x8x8 Matmul 65.0 ms by the
// number of Specs alone, 60.4 with four items a warp, 64.0 with one, 68.6 with sixteen; 16x16 Move 8.4,
// 8.8, 9.8 and 9.1, which is why such Specs keep to the number alone.
__device__ __forceinline__ uint32_t item_log(unsigned long long cells, uint32_t n_late, uint32_t n, uint32_t gwarps) {
  const unsigned long long share = (n_late > 16u ? 128ull : max(128ull, cells / 4)) * n / gwarps;
  return share >= MRL_ITEM_CELLS ? 5u : (share < 32u ? 0u : 26u - __clz((uint32_t)share));
}
// An item's first cell, and its size; first_cell has the size's log in bits 1 to 3 (bit 0: the grid is new).
__device__ __forceinline__ uint32_t item_first(const WorkItem& it) { return it.first_cell & ~31u; }
__device__ __forceinline__ uint32_t item_cells(const WorkItem& it) { return 32u << ((it.first_cell >> 1) & 7u); }

// One pass over the records of a Spec, a record per lane: the breakpoints of the records whose children
// all lie in finished stages (they come first), the corner of those, and of the others with nothing
// known about same-stage children.
__device__ __noinline__ uint4 scan_records(const StageArgs& a, uint32_t lo, const uint2 cl, uint32_t& early, uint32_t& late, uint32_t& n_late,
                                              uint32_t lane) {
  uint4 r = make_uint4(1u, 1u, 1u, 1u);
  early = late = MRL_NEVER4;
  n_late = 0;
  #pragma unroll 1
  for (uint32_t c0 = 0; c0 < cl.y; c0 += 32) {
    bool l = false;
    if (c0 + lane < cl.y) {
      const uint4* const rec = reinterpret_cast<const uint4*>(&a.cands[cl.x + c0 + lane]);
      const uint4 c = __ldg(rec), b = __ldg(rec + 1);
      l = is_late(c);
      const uint32_t q = record_corner(a, lo, c, b, false);
      if (l) late = __vminu4(late, q);
      else {
        early = __vminu4(early, q);
        record_breakpoints(a, lo, c, b, r);
      }
    }
    n_late += __popc(__ballot_sync(0xFFFFFFFFu, l));
  }
  early = warp_min4(early);
  if (n_late) late = warp_min4(late);
  return warp_or(r);
}

// Phase 1.
__device__ __noinline__ void phase_records(const StageArgs& a, StageCtl* sc, uint32_t lo, uint32_t hi, uint32_t gwarp, uint32_t gwarps, uint32_t stage) {
  const uint32_t lane = threadIdx.x & 31;
  #pragma unroll 1
  for (uint32_t i = lo + gwarp; i < hi; i += gwarps) {
    if (!computed_here(a, i)) {
      if (lane == 0) a.rmask[i] = make_uint4(0, 0, 0, 0);   // another rank's Spec: zero until the exchange
      continue;
    }
    uint32_t early, late, n_late;
    const uint4 r = scan_records(a, lo, *reinterpret_cast<const uint2*>(&a.hdrs[i].cand_off), early, late, n_late, lane);
    if (lane == 0) {
      StageSpec& s = a.sspec[i - lo];
      s.emask = r;
      s.corner = early;
      s.n_late = n_late;
      uint32_t bound = __vminu4(early, late);
      if (__vcmpgtu4(bound, a.top_pack)) bound = MRL_NEVER4;   // no limits inside the lattice reach it
      a.minsat[i] = bound;
      if (n_late) sc->any_late = stage + 1;   // every writer of a stage stores the same value
    }
  }
}

// Rows and work items for the grids of up to 32 Specs, one per lane (`cells` 0: none), by one warp:
// the lane's first row, and items at the end of the list. What does not fit is counted and left out;
// the totals are checked behind the next barrier.
__device__ __forceinline__ unsigned long long place_grids(const StageArgs& a, unsigned long long* row_cursor, uint32_t* item_cursor, uint32_t spec, unsigned long long cells,
                                                          unsigned long long item_cells_of, uint32_t log, uint32_t flag, uint32_t lane) {
  unsigned long long inc = cells;
  uint32_t items = (uint32_t)((item_cells_of + (32u << log) - 1) >> (5u + log)), iinc = items;
  flag |= log << 1;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
    const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, iinc, o);
    if (lane >= (uint32_t)o) { inc += t; iinc += u; }
  }
  unsigned long long row0 = 0;
  uint32_t item0 = 0;
  if (lane == 31) {
    if (inc) row0 = atomicAdd(row_cursor, inc);
    if (iinc) item0 = atomicAdd(item_cursor, iinc);
  }
  row0 = __shfl_sync(0xFFFFFFFFu, row0, 31);
  item0 = __shfl_sync(0xFFFFFFFFu, item0, 31);
  uint32_t todo = __ballot_sync(0xFFFFFFFFu, items != 0);
  #pragma unroll 1
  while (todo) {
    const uint32_t src = __ffs(todo) - 1;
    todo &= todo - 1;
    const uint32_t n = __shfl_sync(0xFFFFFFFFu, items, src), at = item0 + __shfl_sync(0xFFFFFFFFu, iinc, src) - n;
    const uint32_t sp = __shfl_sync(0xFFFFFFFFu, spec, src), fl = __shfl_sync(0xFFFFFFFFu, flag, src);
    #pragma unroll 1
    for (uint32_t w = lane; w < n; w += 32)
      if (at + w < a.item_cap) {
        WorkItem it;
        it.spec = sp;
        it.first_cell = (w * item_cells(WorkItem{0, fl})) | fl;
        a.items[at + w] = it;
      }
  }
  return row0 + inc - cells;
}

// Phase 2: the final corner (records with a same-stage child again, with that child's bound), the grid
// of the unordered phase, its rows and work items.
__device__ __noinline__ void phase_place_early(const StageArgs& a, StageCtl* sc, uint32_t lo, uint32_t hi, uint32_t gwarp, uint32_t gwarps, bool any_late) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t G = group_size(hi - lo, gwarps);
  #pragma unroll 1
  for (uint32_t base = lo + gwarp * G; base < hi; base += gwarps * G) {
    const uint32_t i = base + lane;
    const bool mine = lane < G && i < hi && computed_here(a, i);
    uint32_t corner = MRL_NEVER4, n_late = 0;
    uint4 m = make_uint4(1u, 1u, 1u, 1u);
    if (mine) {
      const StageSpec& s = a.sspec[i - lo];
      m = s.emask;
      corner = s.corner;
      n_late = s.n_late;
    }
    uint32_t todo = any_late ? __ballot_sync(0xFFFFFFFFu, n_late != 0) : 0u;
    #pragma unroll 1
    while (todo) {
      const uint32_t src = __ffs(todo) - 1;
      todo &= todo - 1;
      const uint32_t n = __shfl_sync(0xFFFFFFFFu, n_late, src);
      const uint2 cl = *reinterpret_cast<const uint2*>(&a.hdrs[base + src].cand_off);
      uint32_t q = MRL_NEVER4;
      #pragma unroll 1
      for (uint32_t c = lane; c < n; c += 32) {
        const uint4* const rec = reinterpret_cast<const uint4*>(&a.cands[cl.x + cl.y - 1 - c]);
        q = __vminu4(q, record_corner(a, lo, __ldg(rec), __ldg(rec + 1), true));
      }
      q = warp_min4(q);
      if (lane == src) corner = __vminu4(corner, q);
    }
    unsigned long long cells = 0;
    if (mine) {
      if (__vcmpgtu4(corner, a.top_pack)) corner = MRL_NEVER4;
      m = clip_at_corner(m, corner);
      cells = cells_of(m);
    }
    const unsigned long long row = place_grids(a, &sc->rows_early, &sc->n_items_early, i, cells, cells, item_log(cells, n_late, hi - lo, gwarps), 0, lane);
    if (mine) {
      StageSpec& s = a.sspec[i - lo];
      s.emask = m;
      s.corner = corner;
      s.erow = row;
      a.rmask[i] = make_uint4(1u, 1u, 1u, 1u);
    }
  }
}

// Phase 5 (and once more per further pass): the grid the records with a same-stage child are solved
// on: the real breakpoints of what the unordered phase found (first pass: they are in rmask), the
// breakpoints of those records, and for their same-stage children the breakpoints in rmask - first
// pass: of what the unordered phase found for the child; later passes: found real by the pass
// before. Grids only grow; one that grew gets new rows, and its old ones are remembered.
// A Spec without such records is finished: its grid is that of the unordered phase.
__device__ __noinline__ void phase_place_late(const StageArgs& a, StageCtl* sc, uint32_t lo, uint32_t hi, uint32_t gwarp, uint32_t gwarps, uint32_t pass) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t G = group_size(hi - lo, gwarps);
  #pragma unroll 1
  for (uint32_t base = lo + gwarp * G; base < hi; base += gwarps * G) {
    const uint32_t i = base + lane;
    const bool mine = lane < G && i < hi && computed_here(a, i);
    uint32_t n_late = 0, corner = 0;
    uint4 old = make_uint4(0, 0, 0, 0);
    if (mine) {
      const StageSpec& s = a.sspec[i - lo];
      n_late = s.n_late;
      corner = s.corner;
      old = pass ? *reinterpret_cast<const uint4*>(&a.hdrs[i]) : a.rmask[i];
      if (!pass) a.changed[0][i - lo] = a.changed[1][i - lo] = a.changed[2][i - lo] = make_uint4(0, 0, 0, 0);
      if (!pass && !n_late) {
        *reinterpret_cast<uint4*>(&a.hdrs[i]) = s.emask;
        a.hdrs[i].row_base = (a.temp_cap + s.erow) | MRL_TEMP_FLAG;
      }
    }
    uint4 nm = old;
    uint32_t todo = __ballot_sync(0xFFFFFFFFu, n_late != 0);
    #pragma unroll 1
    while (todo) {
      const uint32_t src = __ffs(todo) - 1;
      todo &= todo - 1;
      const uint32_t n = __shfl_sync(0xFFFFFFFFu, n_late, src);
      const uint2 cl = *reinterpret_cast<const uint2*>(&a.hdrs[base + src].cand_off);
      uint4 r = make_uint4(0, 0, 0, 0);
      #pragma unroll 1
      for (uint32_t c = lane; c < n; c += 32) {
        const uint4* const rec = reinterpret_cast<const uint4*>(&a.cands[cl.x + cl.y - 1 - c]);
        record_breakpoints(a, lo, __ldg(rec), __ldg(rec + 1), r);
      }
      r = warp_or(r);
      if (lane == src) { nm.x |= r.x; nm.y |= r.y; nm.z |= r.z; nm.w |= r.w; }
    }
    bool fresh = false;
    unsigned long long cells = 0;
    if (n_late) {
      nm = clip_at_corner(nm, corner);
      fresh = !pass || nm.x != old.x || nm.y != old.y || nm.z != old.z || nm.w != old.w;
      cells = cells_of(nm);
    }
    const unsigned long long row = place_grids(a, &sc->rows_late, &sc->n_items, i, fresh ? cells : 0ull, cells, item_log(cells, n_late, hi - lo, gwarps), fresh ? 1u : 0u, lane);
    if (fresh) {
      StageSpec& s = a.sspec[i - lo];
      s.old_mask = old;
      s.old_row = pass ? a.hdrs[i].row_base : 0ull;
      *reinterpret_cast<uint4*>(&a.hdrs[i]) = nm;
      a.hdrs[i].row_base = row | MRL_TEMP_FLAG;
    }
    if (pass && n_late) a.sspec[i - lo].dirty = fresh ? 1u : 0u;
  }
}

// After a pass: does any grid lack a (shifted) real breakpoint of a same-stage child?
__device__ __noinline__ void phase_check_grids(const StageArgs& a, StageCtl* sc, uint32_t lo, uint32_t hi, uint32_t gwarp, uint32_t gwarps, uint32_t pass) {
  const uint32_t lane = threadIdx.x & 31;
  #pragma unroll 1
  for (uint32_t i = lo + gwarp; i < hi; i += gwarps) {
    if (!computed_here(a, i)) continue;
    const uint32_t n = a.sspec[i - lo].n_late;
    if (!n) continue;
    const uint2 cl = *reinterpret_cast<const uint2*>(&a.hdrs[i].cand_off);
    uint4 r = make_uint4(0, 0, 0, 0);
    #pragma unroll 1
    for (uint32_t c = lane; c < n; c += 32) {
      const uint4* const rec = reinterpret_cast<const uint4*>(&a.cands[cl.x + cl.y - 1 - c]);
      record_breakpoints(a, lo, __ldg(rec), __ldg(rec + 1), r);
    }
    const uint4 m = *reinterpret_cast<const uint4*>(&a.hdrs[i]);
    const uint32_t corner = a.sspec[i - lo].corner;
    // what the grid lacks above its corner (below it nothing is kept)
    const uint32_t k0 = corner_of(corner, 0), k1 = corner_of(corner, 1), k2 = corner_of(corner, 2), k3 = corner_of(corner, 3);
    const bool lacks = k0 != MRL_NEVER && (((r.x & ~m.x) >> k0) | ((r.y & ~m.y) >> k1) | ((r.z & ~m.z) >> k2) | ((r.w & ~m.w) >> k3));
    if (lacks) sc->grew = pass + 1;   // every writer of a pass stores the same value
  }
}

// Step 2: the candidates whose children all lie in earlier stages, for every cell of every
// Spec's grid of the unordered phase. No order is needed. A warp takes a work item (up to MRL_ITEM_CELLS cells of one
// Spec) at a time as it finishes others. Per item it first stages the Spec's records and the
// headers of their children in shared memory, one record per lane, so that the chain record ->
// child header -> child row costs two round trips per batch of records instead of two per record;
// then its lanes take 32 cells at a time and walk the staged records together, and the only
// global loads left in that loop are the child rows.
struct HotArgs {   // what the solve phases read, by value: registers instead of the argument block
  const SpecHdr* hdrs;
  const CandRec* cands;
  MrlRow* rows;
  MrlRow* temp;
  unsigned long long temp_cap;   // the grids of the unordered phase start here
  StageSpec* sspec;              // already offset: indexed by Spec id
  const WorkItem* items;
  uint32_t n_items;
  uint32_t* next_item;
};

constexpr int kBatch = 16;   // records staged at a time
struct StagedRec {           // a record with what the row lookups of its children need
  uint4 rec;                 // action | kind << 16 | nchild << 24, imm, level | thr << 8 | peak << 16, units
  uint4 mask[3];
  const MrlRow* grid[3];     // per child: the first row of its grid, in the table or in the working rows
  uint32_t stride[3][3];     // per child: rows per step in memories 1, 2, 3 of its grid
  uint8_t in_temp[4];        // per child: its grid lies in the working rows (it may change during a sweep)
};
static_assert(sizeof(StagedRec) == 128, "staged record");

// What the lookups of one child need, into its slot of a staged record.
__device__ __forceinline__ void stage_child(StagedRec& s, uint32_t j, const uint4 m, const MrlRow* grid, bool in_temp) {
  s.mask[j] = m;
  s.grid[j] = grid;
  s.in_temp[j] = in_temp ? 1 : 0;
  const uint32_t n0 = __popc(m.x), n1 = __popc(m.y), n2 = __popc(m.z);
  s.stride[j][0] = n0;
  s.stride[j][1] = n0 * n1;
  s.stride[j][2] = n0 * n1 * n2;
}
// row_of with the child's header and strides at hand.
__device__ __forceinline__ const MrlRow* staged_row(const StagedRec& s, uint32_t j, uint32_t b0, uint32_t b1, uint32_t b2, uint32_t b3) {
  const uint4 m = s.mask[j];
  const uint32_t i0 = __popc(m.x & b0) - 1, i1 = __popc(m.y & b1) - 1, i2 = __popc(m.z & b2) - 1, i3 = __popc(m.w & b3) - 1;
  const uint32_t off = i3 * s.stride[j][2] + i2 * s.stride[j][1] + i1 * s.stride[j][0] + i0;   // cells per Spec < 2^32
  return s.grid[j] + off;
}

// The lattice code of every slot of a grid, memory after memory, for the lanes of a warp to look
// up instead of counting bits (a grid has at most 17 + 17 + 12 + 27 slots).
constexpr int kMaxSlots = 80;
constexpr int kMaxAffected = 26;   // more: every cell is solved again
struct WarpScratch {         // a warp's shared memory in the solve phases
  StagedRec staged[kBatch];
  uint4 affected[kMaxAffected];      // sweeps: per changed child the parent's codes that read a changed slot of it
  uint32_t who[32];                  // record (from the end) | child << 16 | position among such records << 20
  uint32_t queue[64];                // sweeps: cells to solve again, as packed slots
  uint16_t reads[64];                // ... and which of the staged records read something that changed there
  union {
    uint32_t bound[kBatch];          // per staged record: no cell of the item gets a main cost below this from it
    uint32_t listed[kBatch];         // or, in later sweeps, the records (from the end) with a changed child
  };
  uint8_t order[kBatch];             // the staged records that can apply, by that bound
  uint8_t codes[kMaxSlots];
};
// With the static shared memory 100 KB a block, which leaves L1 156 KB of an SM; 132 KB is the next step
// (size 8 u32: 2 % slower).
static_assert(sizeof(WarpScratch) == 3136, "warp scratch");

__device__ __forceinline__ void stage_slot_codes(uint8_t* codes, const uint4 m, uint32_t n0, uint32_t n1, uint32_t n2, uint32_t n3,
                                                 uint32_t lane) {
  __syncwarp();   // the previous item's codes have been read by every lane
  #pragma unroll 1
  for (uint32_t t = lane; t < n0 + n1 + n2 + n3; t += 32) {
    uint32_t mk = m.x, slot = t;
    if (slot >= n0) { slot -= n0; mk = m.y; if (slot >= n1) { slot -= n1; mk = m.z; if (slot >= n2) { slot -= n2; mk = m.w; } } }
    codes[t] = (uint8_t)nth_set_bit(mk, slot);
  }
  __syncwarp();
}

// Whole-row accesses to working rows that other warps may be writing at the same time: one
// 128-bit access each, so a reader sees a row either before or after an update, never a mix.
__device__ __forceinline__ uint4 ld_row_shared(const MrlRow* p) {
  unsigned long long lo, hi;
  asm volatile("{\n\t.reg .b128 q;\n\tld.relaxed.gpu.global.b128 q, [%2];\n\tmov.b128 {%0, %1}, q;\n\t}"
               : "=l"(lo), "=l"(hi) : "l"(p) : "memory");
  return make_uint4((uint32_t)lo, (uint32_t)(lo >> 32), (uint32_t)hi, (uint32_t)(hi >> 32));
}
__device__ __forceinline__ void st_row_shared(MrlRow* p, const uint4 v) {
  const unsigned long long lo = v.x | ((unsigned long long)v.y << 32), hi = v.z | ((unsigned long long)v.w << 32);
  asm volatile("{\n\t.reg .b128 q;\n\tmov.b128 q, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], q;\n\t}"
               :: "l"(p), "l"(lo), "l"(hi) : "memory");
}
__device__ __forceinline__ uint4 ld_row(const MrlRow* p) { return *reinterpret_cast<const uint4*>(p); }

// A staged record at one limits point; eval_candidate with the record and the child headers
// already at hand. kMoving: a child's rows may change while this runs. Rows are read with plain
// loads even where they are final: a launch may hold several stages, so they may have been written
// earlier in it, and the read-only path does not see that.
template <bool kMoving>
__device__ __forceinline__ void eval_staged(const StagedRec& s, uint32_t cpack, uint32_t bm0, uint32_t bm1, uint32_t bm2, uint32_t bm3,
                                            Best& best, Tally& tally) {
  const uint4 a = s.rec;
  const uint32_t action = a.x & 0xFFFFu, kind = (a.x >> 16) & 0xFFu, nchild = a.x >> 24;   // the same in all lanes
  const uint32_t imm = a.y;
  const uint32_t level = a.z & 0xFFu, thr = (a.z >> 8) & 0xFFu, pcode = (a.z >> 16) & 0xFFu;
  const uint32_t units = a.w;
  const uint32_t lv = code_of(cpack, level);
  tally.cands++;
  uint32_t k_main, k_peaks, k_tail;
  if (kind == MRL_CK_LEAF) {
    if (lv < thr) return;
    k_main = imm;
    k_peaks = pcode << peak_shift(level);
    k_tail = (1u << 16) | action;
  } else {
    uint32_t c0 = bm0, c1 = bm1, c2 = bm2, c3 = bm3;
    const uint32_t sh = peak_shift(level);
    if (kind == MRL_CK_MOVE) {
      if (lv < thr) return;
      if (imm > best.main) return;   // a Move costs at least its own base cost
      const uint32_t cb = below(child_code(level, lv, units));
      c0 = (level == 0) ? cb : c0;
      c1 = (level == 1) ? cb : c1;
      c2 = (level == 2) ? cb : c2;
      c3 = (level == 3) ? cb : c3;
    }
    uint4 r[3];
#pragma unroll
    for (int j = 0; j < 3; j++) {
      if ((uint32_t)j < nchild) {
        const MrlRow* const p = staged_row(s, j, c0, c1, c2, c3);
        r[j] = (kMoving && s.in_temp[j]) ? ld_row_shared(p) : ld_row(p);
      } else {
        r[j] = r[0];
      }
    }
    tally.lookups += nchild;
    if (r[0].z == MRL_UNSAT || r[1].z == MRL_UNSAT || r[2].z == MRL_UNSAT) return;
    uint32_t depth;
    if (kind == MRL_CK_LOOP) {
      k_main = sat_mul(r[0].x, imm);
      k_peaks = r[0].y;
      depth = 1u;
    } else {
      k_main = (kind == MRL_CK_MOVE) ? sat_add(imm, r[0].x) : r[0].x;
      if (nchild > 1) k_main = sat_add(k_main, r[1].x);
      if (nchild > 2) k_main = sat_add(k_main, r[2].x);
      if (k_main > best.main) return;
      k_peaks = __vmaxu4(__vmaxu4(r[0].y, r[1].y), r[2].y);
      if (kind == MRL_CK_MOVE) {
        const uint32_t cc = (k_peaks >> sh) & 0xFFu;
        const uint32_t ncode = level < 2 ? units + cc : cache_code_ceil(units + cache_value(cc));
        k_peaks = (k_peaks & ~(0xFFu << sh)) | (ncode << sh);
      }
      depth = min(max(max(r[0].z >> 16, r[1].z >> 16), r[2].z >> 16) + 1u, 255u);
    }
    k_tail = (depth << 16) | action;
  }
  if (key_less(k_main, k_peaks, k_tail, best)) {
    best.main = k_main;
    best.peaks = k_peaks;
    best.tail = k_tail;
  }
}

__device__ __forceinline__ WarpScratch& warp_scratch() {
  extern __shared__ uint4 dyn_smem[];
  return reinterpret_cast<WarpScratch*>(dyn_smem)[threadIdx.x >> 5];
}
__device__ __forceinline__ uint32_t warp_number() { return blockIdx.x * (kStageBlock / 32) + (threadIdx.x >> 5); }
__device__ __forceinline__ uint32_t warp_count() { return gridDim.x * (kStageBlock / 32); }
// Every warp starts with the item of its own number; further items are handed out by a counter (no
// atomics at all when there are fewer items than warps).
__device__ __forceinline__ bool next_item(const HotArgs& a, uint32_t& w, uint32_t lane) {
  const uint32_t gwarps = warp_count();
  if (a.n_items <= gwarps) return false;
  if (lane == 0) w = gwarps + atomicAdd(a.next_item, 1u);
  w = __shfl_sync(0xFFFFFFFFu, w, 0);
  return w < a.n_items;
}
__device__ __forceinline__ void add_tally(const Tally& tally, unsigned long long* cands, unsigned long long* lookups, uint32_t lane) {
  const uint32_t tc = __reduce_add_sync(0xFFFFFFFFu, tally.cands), tl = __reduce_add_sync(0xFFFFFFFFu, tally.lookups);
  if (lane == 0 && (tc | tl)) {
    atomicAdd(cands, (unsigned long long)tc);
    atomicAdd(lookups, (unsigned long long)tl);
  }
}

// Limit codes that no cell of [first, end) exceeds: per memory the largest among them. n: slots per
// memory; z: slots left out at the bottom of each (cells are numbered without them).
__device__ __forceinline__ uint32_t top_codes(const uint8_t* codes, uint32_t first, uint32_t end, uint32_t n0, uint32_t n1, uint32_t n2, uint32_t z0,
                                              uint32_t z1, uint32_t z2, uint32_t z3) {
  uint32_t f0, f1, f2, f3, l0, l1, l2, l3;
  cell_slots(first, n0 - z0, n1 - z1, n2 - z2, f0, f1, f2, f3);
  cell_slots(end - 1, n0 - z0, n1 - z1, n2 - z2, l0, l1, l2, l3);
  const bool same3 = f3 == l3, same2 = same3 && f2 == l2, same1 = same2 && f1 == l1;
  const uint32_t t0 = same1 ? l0 + z0 : n0 - 1, t1 = same2 ? l1 + z1 : n1 - 1, t2 = same3 ? l2 + z2 : n2 - 1, t3 = l3 + z3;
  return codes[t0] | (codes[n0 + t1] << 8) | (codes[n0 + n1 + t2] << 16) | ((uint32_t)codes[n0 + n1 + n2 + t3] << 24);
}

// Lower bounds of the staged records over a run of cells, and the order to try them in. More memory
// never makes an optimum's main cost larger nor loses an implementation, so what a record costs with
// its children read at the run's largest limits bounds it from below at every cell of the run, and one
// whose child has no implementation there, or that does not fit, applies nowhere in it. Cells then
// take the records cheapest bound first and stop where no lane's optimum so far is above the bound
// (ties are evaluated: peaks, depth and action number decide those). kMoving: tables that may change
// while this runs bound nothing. Returns the number of records that can apply.
// Evaluating a record at 32 cells is a hundred instructions and 1.4 gathered rows a lane; of the 59 G
// evaluations of the size-8 u32 fill 22 G are left, and the fill takes 490 ms instead of 639.
template <bool kMoving>
__device__ __noinline__ uint32_t stage_bounds(WarpScratch& ws, uint32_t n_here, uint32_t cmax, uint32_t lane) {
  #pragma unroll 1
  for (uint32_t t = lane; t < kBatch * 4u; t += 32) {   // four lanes per record, one per child and one idle
    const uint32_t r = t >> 2, j = t & 3u;
    uint32_t part = 0, kind = MRL_CK_LEAF, imm = 0;
    bool dead = r >= n_here;
    if (!dead) {
      const StagedRec& s = ws.staged[r];
      const uint4 a = s.rec;
      kind = (a.x >> 16) & 0xFFu;
      imm = a.y;
      const uint32_t nchild = a.x >> 24, level = a.z & 0xFFu, lv = code_of(cmax, level);
      if ((kind == MRL_CK_LEAF || kind == MRL_CK_MOVE) && lv < ((a.z >> 8) & 0xFFu)) {
        dead = true;
      } else if (j < nchild && !(kMoving && s.in_temp[j])) {
        uint32_t c = cmax;
        if (kind == MRL_CK_MOVE) c = (c & ~(0xFFu << (8 * level))) | (child_code(level, lv, a.w) << (8 * level));
        const uint4 row = ld_row(staged_row(s, j, below(code_of(c, 0)), below(code_of(c, 1)), below(code_of(c, 2)), below(code_of(c, 3))));
        dead = row.z == MRL_UNSAT;
        part = row.x;
      }
    }
    part = sat_add(part, __shfl_xor_sync(0xFFFFFFFFu, part, 1));
    part = sat_add(part, __shfl_xor_sync(0xFFFFFFFFu, part, 2));
    const uint32_t any_dead = (__ballot_sync(0xFFFFFFFFu, dead) >> (lane & ~3u)) & 0xFu;
    if (j == 0) {
      ws.bound[r] = kind == MRL_CK_LEAF ? imm : (kind == MRL_CK_LOOP ? sat_mul(part, imm) : (kind == MRL_CK_MOVE ? sat_add(part, imm) : part));
      ws.order[r] = any_dead ? 1 : 0;
    }
  }
  __syncwarp();
  const uint32_t own = lane < kBatch ? ws.bound[lane] : 0u;
  const uint32_t alive = __ballot_sync(0xFFFFFFFFu, lane < kBatch && !ws.order[lane & (kBatch - 1)]);
  uint32_t at = 0;
  #pragma unroll 1
  for (uint32_t rest = alive; rest; rest &= rest - 1) {
    const uint32_t k = __ffs(rest) - 1, b = __shfl_sync(0xFFFFFFFFu, own, k);
    at += b < own || (b == own && k < lane);
  }
  __syncwarp();
  if ((alive >> lane) & 1u) ws.order[at] = (uint8_t)lane;
  __syncwarp();
  return __popc(alive);
}
// From this many cells on the bounds of a run of them are worth their reads (one more dependent read per
// record, against one evaluation per record and 32 cells).
constexpr uint32_t kBoundCells = 64;

// The staged records at the lanes' cells. n: what stage_bounds left of them, or all (bounded = false).
template <bool kMoving>
__device__ __forceinline__ void eval_batch(const WarpScratch& ws, uint32_t n, bool bounded, bool live, uint32_t cpack, uint32_t bm0, uint32_t bm1,
                                           uint32_t bm2, uint32_t bm3, Best& best, Tally& tally) {
  #pragma unroll 1
  for (uint32_t q = 0; q < n; q++) {
    uint32_t r = q;
    bool go = live;
    if (bounded) {
      r = ws.order[q];
      go = live && ws.bound[r] <= best.main;
      if (!__any_sync(0xFFFFFFFFu, go)) break;
    }
    if (go) eval_staged<kMoving>(ws.staged[r], cpack, bm0, bm1, bm2, bm3, best, tally);
  }
}

// The records of a Spec whose children all lie in finished stages, for the cells [first, end) of its
// grid of the unordered phase, by a warp. The grid's slot codes are staged.
__device__ __noinline__ void solve_early_cells(const HotArgs a, WarpScratch& ws, uint32_t cand_off, uint32_t n_early, const uint4 m, uint32_t corner,
                                                  MrlRow* grid, uint32_t first, uint32_t end, Tally& tally, uint32_t lane) {
  StagedRec* const staged = ws.staged;
  const uint8_t* const codes = ws.codes;
  const uint32_t n0 = __popc(m.x), n1 = __popc(m.y), n2 = __popc(m.z);
  const bool bounded = end - first > kBoundCells;
  const uint32_t cmax = bounded ? top_codes(codes, first, end, n0, n1, n2, 0, 0, 0, 0) : 0u;
  uint32_t b0 = 0;
  do {
    // stage the next records, and the headers of their children, one (record, child) per lane
    const uint32_t n_here = min((uint32_t)kBatch, n_early - b0);
    __syncwarp();   // the previous batch has been read by every lane
    if (lane < n_here) staged[lane].rec = __ldg(reinterpret_cast<const uint4*>(&a.cands[cand_off + b0 + lane]));
    __syncwarp();
    #pragma unroll 1
    for (uint32_t t = lane; t < n_here * 3u; t += 32) {
      const uint32_t r = t / 3u, j = t - r * 3u;
      if (j < (staged[r].rec.x >> 24)) {
        const uint32_t child = __ldg(&a.cands[cand_off + b0 + r].child[j]);
        stage_child(staged[r], j, *reinterpret_cast<const uint4*>(&a.hdrs[child]), a.rows + a.hdrs[child].row_base, false);
      }
    }
    __syncwarp();
    const uint32_t n_apply = bounded ? stage_bounds<false>(ws, n_here, cmax, lane) : n_here;
    #pragma unroll 1
    for (uint32_t c0 = first; c0 < end; c0 += 32) {
      const uint32_t cell = c0 + lane;
      const bool valid = cell < end;
      uint32_t s0, s1, s2, s3;
      cell_slots(valid ? cell : 0u, n0, n1, n2, s0, s1, s2, s3);
      const uint32_t k0 = codes[s0], k1 = codes[n0 + s1], k2 = codes[n0 + n1 + s2], k3 = codes[n0 + n1 + n2 + s3];
      const uint32_t cpack = k0 | (k1 << 8) | (k2 << 16) | (k3 << 24);
      const bool live = valid && !below_corner(corner, cpack);
      Best best = {MRL_UNSAT, MRL_UNSAT, MRL_UNSAT};
      if (!__any_sync(0xFFFFFFFFu, live)) {
        if (valid && b0 == 0) *reinterpret_cast<uint4*>(grid + cell) = make_uint4(best.main, best.peaks, best.tail, 0u);
        continue;
      }
      if (b0 && live) {   // what the earlier batches found
        const uint4 r = ld_row(grid + cell);
        best.main = r.x; best.peaks = r.y; best.tail = r.z;
      }
      eval_batch<false>(ws, n_apply, bounded, live, cpack, below(k0), below(k1), below(k2), below(k3), best, tally);
      if (valid && (b0 == 0 || live)) *reinterpret_cast<uint4*>(grid + cell) = make_uint4(best.main, best.peaks, best.tail, 0u);
    }
    b0 += n_here;
  } while (b0 < n_early);
}

__device__ __noinline__ void phase_early(const HotArgs a, unsigned long long* block_stats) {
  const uint32_t lane = threadIdx.x & 31;
  WarpScratch& ws = warp_scratch();
  Tally tally = {0, 0};
  uint32_t w = warp_number();
  if (w < a.n_items)
#pragma unroll 1
  do {
    const WorkItem it = a.items[w];
    const StageSpec& sp = a.sspec[it.spec];
    const uint4 m = sp.emask;
    const uint2 cl = *reinterpret_cast<const uint2*>(&a.hdrs[it.spec].cand_off);
    stage_slot_codes(ws.codes, m, __popc(m.x), __popc(m.y), __popc(m.z), __popc(m.w), lane);
    solve_early_cells(a, ws, cl.x, cl.y - sp.n_late, m, sp.corner, a.temp + a.temp_cap + sp.erow, item_first(it),
                      min((uint32_t)cells_of(m), item_first(it) + item_cells(it)), tally, lane);
  } while (next_item(a, w, lane));
  add_tally(tally, &block_stats[0], &block_stats[1], lane);
}

// Step 4, relaxation sweeps: the records with a child in the Spec's own stage (relayout Moves). Such
// a child is read at limits reduced by what the Move allocates, so the dependencies between cells
// form no cycle and the system "cell = best of its candidates at its children's values" has exactly
// one solution. A sweep recomputes cells from what the unordered phase found at their limits and all
// their same-stage records at the children's current values, in place, while other warps read and
// write their own cells. (Keeping the better of the old and the new value instead of recomputing
// would be wrong: a child that improves can make the parent's peaks or depth worse.) Which cells:
//   first pass, first sweep   all of them, their same-stage children at what the unordered phase
//                             found for those - tables that do not change during the sweep, so the
//                             working rows need no initial values
//   later pass, first sweep   of the grids that grew (their cells hold the old grid's values, copied
//                             at their limits), those that start at a new breakpoint in some memory:
//                             the others read the same children at the same limits as before
//   every other sweep         those that read a slot of a child which the sweep before changed. A
//                             sweep leaves, per Spec and memory, the codes of the slots it changed a
//                             cell of; a cell is solved again when its limits at some child fall into
//                             such slots in all four memories - from the records with such children
//                             alone, where a batch holds them (the size-8 u32 fill's sweeps after the
//                             first: 120 ms with all records, 80 so).
// Every cell is thus consistent with its children when a sweep changes nothing anywhere: it was
// solved after its children last changed, or nothing it reads has changed. At size 8 this took the
// sweeps after the first from 459 ms (whole Specs solved again when a child changed anywhere) to a
// small part of that.
// The records come dearest first and are staged from the end, so the cheapest Move is tried first.
enum { SWEEP_ALL = 0, SWEEP_NEW = 1, SWEEP_CHANGED = 2 };

template <bool kAll>
__device__ __forceinline__ void stage_late_batch(const HotArgs& a, uint32_t lo, StagedRec* staged, uint32_t last_rec, uint32_t n_here, uint32_t lane,
                                                 const uint32_t* listed = nullptr) {
  __syncwarp();   // the previous batch has been read by every lane
  if (lane < n_here) staged[lane].rec = __ldg(reinterpret_cast<const uint4*>(&a.cands[last_rec - (listed ? listed[lane] : lane)]));
  __syncwarp();
  #pragma unroll 1
  for (uint32_t t = lane; t < n_here * 3u; t += 32) {
    const uint32_t r = t / 3u, j = t - r * 3u;
    if (j < (staged[r].rec.x >> 24)) {
      const uint32_t child = __ldg(&a.cands[last_rec - (listed ? listed[r] : r)].child[j]);
      if (kAll && child >= lo) {
        stage_child(staged[r], j, a.sspec[child].emask, a.temp + a.temp_cap + a.sspec[child].erow, false);
      } else {
        const unsigned long long base = a.hdrs[child].row_base;
        stage_child(staged[r], j, *reinterpret_cast<const uint4*>(&a.hdrs[child]), row_at(a.rows, a.temp, base), (base & MRL_TEMP_FLAG) != 0);
      }
    }
  }
  __syncwarp();
}

// The parent's codes in memory k whose lookups of a child end in one of the child's slots `changed`
// (a mask of the slots' codes). parent, child: masks of the two grids.
__device__ __forceinline__ uint32_t codes_reading(uint32_t parent, uint32_t child, uint32_t changed, bool shifted, uint32_t level, uint32_t thr,
                                                  uint32_t units) {
  uint32_t out = 0;
  #pragma unroll 1
  while (parent) {
    const uint32_t p = __ffs(parent) - 1;
    parent &= parent - 1;
    if (shifted && p < thr) continue;   // the Move does not fit
    const uint32_t q = shifted ? child_code(level, p, units) : p;
    const uint32_t slot = 31 - __clz(child & below(q));   // bit 0 is always set
    if ((changed >> slot) & 1u) out |= 1u << p;
  }
  return out;
}

template <bool kAll>
__device__ __noinline__ void phase_sweep(const HotArgs a, int mode, uint32_t lo, const uint4* changed_before, uint4* changed_now, uint32_t sweep, uint32_t* any_changed,
                                         unsigned long long* block_stats) {
  const uint32_t lane = threadIdx.x & 31;
  WarpScratch& ws = warp_scratch();
  StagedRec* const staged = ws.staged;
  const uint8_t* const codes = ws.codes;
  Tally tally = {0, 0};
  uint32_t w = warp_number();
  if (w < a.n_items)
#pragma unroll 1
  do {
    const WorkItem it = a.items[w];
    const uint32_t i = it.spec, first_cell = item_first(it);
    if (!kAll && mode == SWEEP_NEW && !(it.first_cell & 1u)) continue;   // the grid did not grow
    const uint2 cl = *reinterpret_cast<const uint2*>(&a.hdrs[i].cand_off);
    const uint32_t n_late = a.sspec[i].n_late, last = cl.x + cl.y - 1;   // the records with a same-stage child are the last ones
    const uint4 m = *reinterpret_cast<const uint4*>(&a.hdrs[i]);
    uint32_t n_aff = 0, n_listed = 0;   // n_listed: records with a changed child, if a batch holds them
    if (!kAll && mode == SWEEP_NEW) {
      if (lane == 0) {
        const uint4 om = a.sspec[i].old_mask;
        ws.affected[0] = make_uint4(m.x & ~om.x, m.y & ~om.y, m.z & ~om.z, m.w & ~om.w);
      }
      __syncwarp();
    }
    if (!kAll && mode == SWEEP_CHANGED) {
      // children that the sweep before changed
      __syncwarp();   // the previous item's list has been read by every lane
      #pragma unroll 1
      for (uint32_t t0 = 0; t0 < n_late * 3u; t0 += 32) {
        const uint32_t t = t0 + lane, r = t / 3u, j = t - r * 3u;
        bool hit = false;
        if (r < n_late) {
          const CandRec* const rec = &a.cands[last - r];
          if (j < (__ldg(reinterpret_cast<const uint32_t*>(rec)) >> 24)) {
            const uint32_t child = __ldg(&rec->child[j]);
            hit = child >= lo && changed_before[child - lo].x != 0;
          }
        }
        const uint32_t hits = __ballot_sync(0xFFFFFFFFu, hit);
        const uint32_t at = n_aff + __popc(hits & ((1u << lane) - 1u));
        if (hit && at < kMaxAffected) ws.who[at] = r | (j << 16);
        n_aff += __popc(hits);
      }
      if (!n_aff) continue;
      __syncwarp();
      // per such child and memory, the codes of this grid that read one of its changed slots
      if (n_aff <= kMaxAffected) {
        const uint32_t r_own = lane < n_aff ? ws.who[lane] & 0xFFFFu : 0xFFFFu;
        const uint32_t r_prev = __shfl_up_sync(0xFFFFFFFFu, r_own, 1);
        const bool fresh = lane < n_aff && (lane == 0 || r_prev != r_own);   // a record's children follow one another
        const uint32_t firsts = __ballot_sync(0xFFFFFFFFu, fresh), at = __popc(firsts & (0xFFFFFFFFu >> (31 - lane))) - 1;
        if (__popc(firsts) <= kBatch) {
          n_listed = __popc(firsts);
          if (fresh) ws.listed[at] = r_own;
        }
        __syncwarp();
        if (lane < n_aff) ws.who[lane] |= at << 20;
        __syncwarp();
        #pragma unroll 1
        for (uint32_t t = lane; t < n_aff * 4u; t += 32) {
          const uint32_t k = t & 3u, r = ws.who[t >> 2] & 0xFFFFu, j = (ws.who[t >> 2] >> 16) & 0xFu;
          const CandRec* const rec = &a.cands[last - r];
          const uint4 c = __ldg(reinterpret_cast<const uint4*>(rec));
          const uint32_t child = __ldg(&rec->child[j]), level = c.z & 0xFFu;
          const uint4 cm = *reinterpret_cast<const uint4*>(&a.hdrs[child]);
          const uint4 ch = changed_before[child - lo];
          reinterpret_cast<uint32_t*>(&ws.affected[t >> 2])[k] =
              codes_reading(sel4(m.x, m.y, m.z, m.w, k), sel4(cm.x, cm.y, cm.z, cm.w, k), sel4(ch.x, ch.y, ch.z, ch.w, k), k == level, level,
                            (c.z >> 8) & 0xFFu, c.w);
        }
      }
      __syncwarp();
    }
    if (lane == 0) atomicAdd(&block_stats[4], 1ull);
    MrlRow* const grid = a.temp + (a.hdrs[i].row_base & ~MRL_TEMP_FLAG);
    const uint4 em = a.sspec[i].emask;   // where the unordered phase left its result
    const MrlRow* const egrid = a.temp + a.temp_cap + a.sspec[i].erow;
    const uint32_t n0 = __popc(m.x), n1 = __popc(m.y), n2 = __popc(m.z), n3 = __popc(m.w);
    const uint32_t cells = n0 * n1 * n2 * n3;
    const uint32_t corner = a.sspec[i].corner;
    // Grids are clipped at the corner, so the cells below it are exactly those in slot 0 of a
    // clipped memory; they stay unsatisfiable and are left out: the lanes walk the live cells
    // only. The item's share of them: its range of all cells, scaled (the items of a Spec tile
    // its cells, so the scaled ranges tile the live ones).
    const bool none = corner_of(corner, 0) == MRL_NEVER;
    const uint32_t z0 = corner_of(corner, 0) ? 1u : 0u, z1 = corner_of(corner, 1) ? 1u : 0u, z2 = corner_of(corner, 2) ? 1u : 0u,
                   z3 = corner_of(corner, 3) ? 1u : 0u;
    const uint32_t v0 = n0 - z0, v1 = n1 - z1, v2 = n2 - z2, v3 = n3 - z3;
    const uint32_t live_cells = none ? 0u : v0 * v1 * v2 * v3;
    const uint32_t c_hi = min(cells, first_cell + item_cells(it));
    uint32_t l_begin = 0, l_end = live_cells;
    if (cells > item_cells(it)) {   // several items
      l_begin = (uint32_t)((unsigned long long)live_cells * first_cell / cells);
      l_end = (uint32_t)((unsigned long long)live_cells * c_hi / cells);
    }
    if (kAll) {   // the cells below the corner
      #pragma unroll 1
      for (uint32_t cell = first_cell + lane; cell < c_hi; cell += 32) {
        uint32_t s0, s1, s2, s3;
        cell_slots(cell, n0, n1, n2, s0, s1, s2, s3);
        if (none || s0 < z0 || s1 < z1 || s2 < z2 || s3 < z3) *reinterpret_cast<uint4*>(grid + cell) = make_uint4(MRL_UNSAT, MRL_UNSAT, MRL_UNSAT, 0u);
      }
    }
    if (l_begin == l_end) continue;
    const bool single = n_late <= (uint32_t)kBatch;   // all records staged once for the whole item
    stage_slot_codes(ws.codes, m, n0, n1, n2, n3, lane);
    const bool bounded = l_end - l_begin > kBoundCells && (kAll || single) && !n_listed;
    const uint32_t cmax = bounded ? top_codes(codes, l_begin, l_end, n0, n1, n2, z0, z1, z2, z3) : 0u;
    uint4 ch = make_uint4(0, 0, 0, 0);   // codes of the slots of the cells that change
    if (kAll) {
      // every cell, one batch of records after the other: nothing reads the working rows meanwhile, so
      // they hold what the batches so far have found
#pragma unroll 1
      for (uint32_t b = 0; b < n_late; b += kBatch) {
        const uint32_t n_here = min((uint32_t)kBatch, n_late - b);
        stage_late_batch<true>(a, lo, staged, last - b, n_here, lane);
        const uint32_t n_apply = bounded ? stage_bounds<false>(ws, n_here, cmax, lane) : n_here;
#pragma unroll 1
        for (uint32_t c0 = l_begin; c0 < l_end; c0 += 32) {
          const bool live = c0 + lane < l_end;
          uint32_t s0, s1, s2, s3;
          cell_slots(live ? c0 + lane : l_begin, v0, v1, v2, s0, s1, s2, s3);
          s0 += z0; s1 += z1; s2 += z2; s3 += z3;
          const uint32_t k0 = codes[s0], k1 = codes[n0 + s1], k2 = codes[n0 + n1 + s2], k3 = codes[n0 + n1 + n2 + s3];
          const uint32_t bm0 = below(k0), bm1 = below(k1), bm2 = below(k2), bm3 = below(k3);
          MrlRow* const at = grid + (((s3 * n2 + s2) * n1 + s1) * n0 + s0);
          const uint32_t i0 = __popc(em.x & bm0) - 1, i1 = __popc(em.y & bm1) - 1, i2 = __popc(em.z & bm2) - 1, i3 = __popc(em.w & bm3) - 1;
          const uint4 f = ld_row(egrid + (((i3 * __popc(em.z) + i2) * __popc(em.y) + i1) * __popc(em.x) + i0));
          const uint4 was = b ? ld_row(at) : f;
          Best best = {was.x, was.y, was.z};
          eval_batch<false>(ws, n_apply, bounded, live, k0 | (k1 << 8) | (k2 << 16) | (k3 << 24), bm0, bm1, bm2, bm3, best, tally);
          if (live) {
            *reinterpret_cast<uint4*>(at) = make_uint4(best.main, best.peaks, best.tail, 0u);
            if (best.main != f.x || best.peaks != f.y || best.tail != f.z) { ch.x |= 1u << k0; ch.y |= 1u << k1; ch.z |= 1u << k2; ch.w |= 1u << k3; }
          }
        }
      }
    } else {
    bool staged_yet = false;
    uint32_t n_apply = n_late;
    uint32_t c0 = l_begin, queued = 0;
#pragma unroll 1
    for (;;) {
      // the next cells to solve, one per lane, collected from those that qualify
      bool live;
      uint32_t slots, reads;
      {
#pragma unroll 1
        while (queued < 32 && c0 < l_end) {
          const bool in = c0 + lane < l_end;
          uint32_t s0, s1, s2, s3;
          cell_slots(in ? c0 + lane : l_begin, v0, v1, v2, s0, s1, s2, s3);
          s0 += z0; s1 += z1; s2 += z2; s3 += z3;
          const uint32_t k0 = codes[s0], k1 = codes[n0 + s1], k2 = codes[n0 + n1 + s2], k3 = codes[n0 + n1 + n2 + s3];
          uint32_t hit = 0;
          if (mode == SWEEP_NEW) {
            const uint4 f = ws.affected[0];
            hit = (f.x >> k0) | (f.y >> k1) | (f.z >> k2) | (f.w >> k3);
          } else if (n_aff > (uint32_t)kMaxAffected) {
            hit = 1;
          } else {
#pragma unroll 1
            for (uint32_t e = 0; e < n_aff; e++) {
              const uint4 f = ws.affected[e];
              hit |= ((f.x >> k0) & (f.y >> k1) & (f.z >> k2) & (f.w >> k3) & 1u) << (ws.who[e] >> 20);
            }
          }
          const bool again = in && (mode == SWEEP_NEW ? hit & 1u : hit);
          const uint32_t who = __ballot_sync(0xFFFFFFFFu, again);
          if (again) {
            const uint32_t at = queued + __popc(who & ((1u << lane) - 1u));
            ws.queue[at] = s0 | (s1 << 8) | (s2 << 16) | (s3 << 24);
            ws.reads[at] = (uint16_t)hit;
          }
          queued += __popc(who);
          c0 += 32;
        }
        if (!queued) break;
        __syncwarp();
        live = lane < queued;
        slots = live ? ws.queue[lane] : (z0 | (z1 << 8) | (z2 << 16) | (z3 << 24));
        reads = live ? ws.reads[lane] : 0u;
        const uint32_t rest_of = ws.queue[32 + lane], rest_reads = ws.reads[32 + lane];
        __syncwarp();
        queued = queued > 32 ? queued - 32 : 0;
        if (lane < queued) {
          ws.queue[lane] = rest_of;
          ws.reads[lane] = (uint16_t)rest_reads;
        }
      }
      if (n_listed) {
        if (!staged_yet) stage_late_batch<false>(a, lo, staged, last, n_listed, lane, ws.listed);
        staged_yet = true;
      } else if (single && !staged_yet) {
        stage_late_batch<false>(a, lo, staged, last, n_late, lane);
        if (bounded) n_apply = stage_bounds<true>(ws, n_late, cmax, lane);
        staged_yet = true;
      }
      const uint32_t s0 = slots & 0xFFu, s1 = (slots >> 8) & 0xFFu, s2 = (slots >> 16) & 0xFFu, s3 = slots >> 24;
      const uint32_t k0 = codes[s0], k1 = codes[n0 + s1], k2 = codes[n0 + n1 + s2], k3 = codes[n0 + n1 + n2 + s3];
      const uint32_t cpack = k0 | (k1 << 8) | (k2 << 16) | (k3 << 24);
      const uint32_t bm0 = below(k0), bm1 = below(k1), bm2 = below(k2), bm3 = below(k3);
      MrlRow* const at = grid + (((s3 * n2 + s2) * n1 + s1) * n0 + s0);
      Best best = {MRL_UNSAT, MRL_UNSAT, MRL_UNSAT};
      uint4 was = make_uint4(MRL_UNSAT, MRL_UNSAT, MRL_UNSAT, 0u);
      if (live) was = ld_row(at);   // only this warp writes the cell in this sweep
      bool whole = live;            // solve it from all its records
      if (n_listed) {
        // The other records cost what they did when the cell was last solved, so the cell's row still is
        // the best of them, unless it came from one of these: then these alone decide as long as they
        // reach the row again, and all records do where they fall short of it.
        const uint32_t any = __reduce_or_sync(0xFFFFFFFFu, reads);
        bool own = false;
#pragma unroll 1
        for (uint32_t rest = any; rest; rest &= rest - 1) {
          const uint32_t r = __ffs(rest) - 1;
          own |= ((reads >> r) & 1u) && (staged[r].rec.x & 0xFFFFu) == (was.z & 0xFFFFu);
        }
        own = own && was.z != MRL_UNSAT;
        if (!own) { best.main = was.x; best.peaks = was.y; best.tail = was.z; }
#pragma unroll 1
        for (uint32_t rest = any; rest; rest &= rest - 1) {
          const uint32_t r = __ffs(rest) - 1;
          if ((reads >> r) & 1u) eval_staged<true>(staged[r], cpack, bm0, bm1, bm2, bm3, best, tally);
        }
        whole = own && key_less(was.x, was.y, was.z, best);
      }
      if (__any_sync(0xFFFFFFFFu, whole)) {
        if (whole) {
          const uint32_t i0 = __popc(em.x & bm0) - 1, i1 = __popc(em.y & bm1) - 1, i2 = __popc(em.z & bm2) - 1, i3 = __popc(em.w & bm3) - 1;
          const uint4 f = ld_row(egrid + (((i3 * __popc(em.z) + i2) * __popc(em.y) + i1) * __popc(em.x) + i0));
          best.main = f.x; best.peaks = f.y; best.tail = f.z;
        }
#pragma unroll 1
        for (uint32_t b = 0; b < n_late; b += kBatch) {
          const uint32_t n_here = min((uint32_t)kBatch, n_late - b);
          if (!single || n_listed) stage_late_batch<false>(a, lo, staged, last - b, n_here, lane);
          eval_batch<true>(ws, single && !n_listed ? n_apply : n_here, bounded, whole, cpack, bm0, bm1, bm2, bm3, best, tally);
        }
        if (n_listed) staged_yet = false;   // the listed ones have been overwritten
      }
      if (live && (best.main != was.x || best.peaks != was.y || best.tail != was.z)) {
        st_row_shared(at, make_uint4(best.main, best.peaks, best.tail, 0u));
        ch.x |= 1u << k0; ch.y |= 1u << k1; ch.z |= 1u << k2; ch.w |= 1u << k3;
      }
    }
    }
    ch = warp_or(ch);
    if (ch.x && lane == 0) {
      uint32_t* const out = reinterpret_cast<uint32_t*>(&changed_now[i - lo]);
      atomicOr(out, ch.x); atomicOr(out + 1, ch.y); atomicOr(out + 2, ch.z); atomicOr(out + 3, ch.w);
      a.sspec[i].dirty = 1;
      *any_changed = sweep;
    }
  } while (next_item(a, w, lane));
  add_tally(tally, &block_stats[2], &block_stats[3], lane);
}

// A further pass: the cells of the grids that grew start from the old grid's values at their limits.
__device__ __noinline__ void phase_refine(const HotArgs a) {
  const uint32_t lane = threadIdx.x & 31;
  uint32_t w = warp_number();
  if (w < a.n_items)
#pragma unroll 1
  do {
    const WorkItem it = a.items[w];
    if (!(it.first_cell & 1u)) continue;
    const uint32_t i = it.spec, first_cell = item_first(it);
    const uint4 m = *reinterpret_cast<const uint4*>(&a.hdrs[i]);
    MrlRow* const grid = a.temp + (a.hdrs[i].row_base & ~MRL_TEMP_FLAG);
    const uint4 om = a.sspec[i].old_mask;
    const unsigned long long obase = a.sspec[i].old_row;
    const uint32_t n0 = __popc(m.x), n1 = __popc(m.y), n2 = __popc(m.z), n3 = __popc(m.w);
    const uint32_t c_end = min(n0 * n1 * n2 * n3, first_cell + item_cells(it));
    #pragma unroll 1
    for (uint32_t cell = first_cell + lane; cell < c_end; cell += 32) {
      uint32_t s0, s1, s2, s3;
      cell_slots(cell, n0, n1, n2, s0, s1, s2, s3);
      const uint32_t k0 = nth_set_bit(m.x, s0), k1 = nth_set_bit(m.y, s1), k2 = nth_set_bit(m.z, s2), k3 = nth_set_bit(m.w, s3);
      *reinterpret_cast<uint4*>(grid + cell) = ld_row(row_of(a.rows, a.temp, om, obase, below(k0), below(k1), below(k2), below(k3)));
    }
  } while (next_item(a, w, lane));
}

// Which breakpoints of a grid are real, from its cells [first, end), by a warp: a breakpoint (memory k,
// code c) is real when some cell starting at c differs from its neighbour one slot lower in k. The
// comparing stops in a memory at codes known to be real. The grid's slot codes are staged.
__device__ __noinline__ uint4 real_breakpoints(const uint8_t* codes, const uint4 m, const MrlRow* grid, uint32_t first, uint32_t end, uint32_t lane) {
  const uint32_t n0 = __popc(m.x), n1 = __popc(m.y), n2 = __popc(m.z);
  const uint32_t st1 = n0, st2 = n0 * n1, st3 = st2 * n2;
  uint4 real = make_uint4(1u, 1u, 1u, 1u);   // the same in all lanes
  #pragma unroll 1
  for (uint32_t c0 = first; c0 < end; c0 += 32) {
    const uint32_t cell = c0 + lane;
    uint4 bits = make_uint4(0, 0, 0, 0);
    if (cell < end) {
      uint32_t s0, s1, s2, s3;
      cell_slots(cell, n0, n1, n2, s0, s1, s2, s3);
      const MrlRow* const p = grid + cell;
      const uint32_t q0 = 1u << codes[s0], q1 = 1u << codes[n0 + s1], q2 = 1u << codes[n0 + n1 + s2], q3 = 1u << codes[n0 + n1 + n2 + s3];
      const bool w0 = s0 && !(real.x & q0), w1 = s1 && !(real.y & q1), w2 = s2 && !(real.z & q2), w3 = s3 && !(real.w & q3);
      if (w0 || w1 || w2 || w3) {
        const uint4 r = ld_row(p);
        uint4 x0 = r, x1 = r, x2 = r, x3 = r;
        if (w0) x0 = ld_row(p - 1);
        if (w1) x1 = ld_row(p - st1);
        if (w2) x2 = ld_row(p - st2);
        if (w3) x3 = ld_row(p - st3);
        if (x0.x != r.x || x0.y != r.y || x0.z != r.z) bits.x = q0;
        if (x1.x != r.x || x1.y != r.y || x1.z != r.z) bits.y = q1;
        if (x2.x != r.x || x2.y != r.y || x2.z != r.z) bits.z = q2;
        if (x3.x != r.x || x3.y != r.y || x3.z != r.z) bits.w = q3;
      }
    }
    bits = warp_or(bits);
    real.x |= bits.x; real.y |= bits.y; real.z |= bits.z; real.w |= bits.w;
  }
  return real;
}

// kEarly: of the grids of the unordered phase, else of the working grids (only_dirty: of those that
// grew or changed).
template <bool kEarly>
__device__ __noinline__ void phase_real_masks(const HotArgs a, uint4* rmask, bool only_dirty) {
  const uint32_t lane = threadIdx.x & 31;
  WarpScratch& ws = warp_scratch();
  uint32_t w = warp_number();
  if (w < a.n_items)
#pragma unroll 1
  do {
    const WorkItem it = a.items[w];
    const uint32_t i = it.spec, first_cell = item_first(it);
    if (only_dirty && !a.sspec[i].dirty) continue;
    const uint4 m = kEarly ? a.sspec[i].emask : *reinterpret_cast<const uint4*>(&a.hdrs[i]);
    const MrlRow* const grid = kEarly ? a.temp + a.temp_cap + a.sspec[i].erow : a.temp + (a.hdrs[i].row_base & ~MRL_TEMP_FLAG);
    stage_slot_codes(ws.codes, m, __popc(m.x), __popc(m.y), __popc(m.z), __popc(m.w), lane);
    const uint4 real = real_breakpoints(ws.codes, m, grid, first_cell, min((uint32_t)cells_of(m), first_cell + item_cells(it)), lane);
    if (lane == 0) {
      uint32_t* const out = reinterpret_cast<uint32_t*>(&rmask[i]);
      if (real.x & ~1u) atomicOr(out, real.x);
      if (real.y & ~1u) atomicOr(out + 1, real.y);
      if (real.z & ~1u) atomicOr(out + 2, real.z);
      if (real.w & ~1u) atomicOr(out + 3, real.w);
    }
  } while (next_item(a, w, lane));
}

// Phases 1 to 4 in one, for the small teams: a warp takes a Spec from its records to the real
// breakpoints of its grid of the unordered phase, without a barrier between. Grids of more than
// kInlineCells cells become work items for the phases proper. The corner is the first round's: a
// weaker bound makes more cells, not other rows.
constexpr uint32_t kInlineCells = 128;
constexpr uint32_t kWarmLines = 960;   // 120 KB
__device__ __noinline__ void phase_early_fused(const StageArgs& a, const HotArgs h, StageCtl* sc, uint32_t lo, uint32_t hi, uint32_t gwarp, uint32_t gwarps,
                                               uint32_t stage, unsigned long long* block_stats) {
  const uint32_t lane = threadIdx.x & 31;
  WarpScratch& ws = warp_scratch();
  Tally tally = {0, 0};
  #pragma unroll 1
  for (uint32_t i = lo + gwarp; i < hi; i += gwarps) {
    if (!computed_here(a, i)) {
      if (lane == 0) a.rmask[i] = make_uint4(0, 0, 0, 0);   // another rank's Spec: zero until the exchange
      continue;
    }
    uint32_t corner, n_late;
    const uint2 cl = *reinterpret_cast<const uint2*>(&a.hdrs[i].cand_off);
    uint4 m;
    {
      uint32_t early, late;
      m = scan_records(a, lo, cl, early, late, n_late, lane);
      corner = __vminu4(early, late);
      if (__vcmpgtu4(corner, a.top_pack)) corner = MRL_NEVER4;   // no limits inside the lattice reach it
    }
    m = clip_at_corner(m, corner);
    const unsigned long long cells = cells_of(m);
    const bool here = cells <= kInlineCells;
    const uint32_t log = item_log(cells, n_late, hi - lo, gwarps);
    const uint32_t n_items = here ? 0u : (uint32_t)((cells + (32u << log) - 1) >> (5u + log));
    unsigned long long row = 0;
    uint32_t item0 = 0;
    if (lane == 0) {
      row = atomicAdd(&sc->rows_early, cells);
      if (n_items) item0 = atomicAdd(&sc->n_items_early, n_items);
    }
    row = __shfl_sync(0xFFFFFFFFu, row, 0);
    item0 = __shfl_sync(0xFFFFFFFFu, item0, 0);
    #pragma unroll 1
    for (uint32_t w = lane; w < n_items; w += 32) {
      const uint32_t at = item0 + w;
      if (at < a.item_cap) {
        WorkItem it;
        it.spec = i;
        it.first_cell = (w << (5u + log)) | (log << 1);
        a.items[at] = it;
      }
    }
    uint4 real = make_uint4(1u, 1u, 1u, 1u);
    if (here && row + cells <= a.temp_cap) {   // (the total is checked behind the barrier)
      MrlRow* const grid = a.temp + a.temp_cap + row;
      stage_slot_codes(ws.codes, m, __popc(m.x), __popc(m.y), __popc(m.z), __popc(m.w), lane);
      solve_early_cells(h, ws, cl.x, cl.y - n_late, m, corner, grid, 0, (uint32_t)cells, tally, lane);
      __syncwarp();   // the lanes' rows, for the others to compare with
      real = real_breakpoints(ws.codes, m, grid, 0, (uint32_t)cells, lane);
    }
    if (lane == 0) {
      StageSpec& s = a.sspec[i - lo];
      s.emask = m;
      s.erow = row;
      s.corner = corner;
      s.n_late = n_late;
      a.rmask[i] = real;
      if (n_late) {
        sc->any_late = stage + 1;   // every writer of a stage stores the same value
      } else {                      // finished: its grid is that of the unordered phase
        *reinterpret_cast<uint4*>(&a.hdrs[i]) = m;
        a.hdrs[i].row_base = (a.temp_cap + row) | MRL_TEMP_FLAG;
      }
    }
  }
  add_tally(tally, &block_stats[0], &block_stats[1], lane);
}

// ---- compaction: working grids -> final table ---------------------------------------------

// The Specs a block counts and compacts: a contiguous part of the stage, so that the places of its
// rows follow from the sums of the blocks before it.
__device__ __forceinline__ void block_specs(uint32_t lo, uint32_t hi, uint32_t& b_lo, uint32_t& b_hi) {
  const uint32_t per = (hi - lo + gridDim.x - 1) / gridDim.x;
  b_lo = min(hi, lo + blockIdx.x * per);
  b_hi = min(hi, b_lo + per);
}

__device__ __forceinline__ unsigned long long block_sum(unsigned long long v) {
  __shared__ unsigned long long part[kStageBlock / 32];
  __shared__ unsigned long long all;
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
  __syncthreads();   // protects the shared values across consecutive calls
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    unsigned long long s = threadIdx.x < kStageBlock / 32 ? part[threadIdx.x] : 0ull;
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, o);
    if (threadIdx.x == 0) all = s;
  }
  __syncthreads();
  return all;
}

// Final cells of this block's Specs, by their real breakpoints.
__device__ __noinline__ void phase_count(const StageArgs& a, uint32_t lo, uint32_t hi) {
  uint32_t b_lo, b_hi;
  block_specs(lo, hi, b_lo, b_hi);
  unsigned long long n = 0;
  #pragma unroll 1
  for (uint32_t i = b_lo + threadIdx.x; i < b_hi; i += kStageBlock) n += cells_of(a.rmask[i]);
  n = block_sum(n);
  if (threadIdx.x == 0) a.block_sums[blockIdx.x] = n;
}

// Copies each Spec's real cells from its grid to its final rows (from first_row on) and repoints the
// header, a warp per Spec. Specs computed by another rank get zero rows (the exchange adds the
// owner's rows onto them). Returns the rows that this block's Specs take.
__device__ __noinline__ unsigned long long phase_compact(const StageArgs& a, uint32_t lo, uint32_t hi, unsigned long long first_row,
                                                         unsigned long long* block_bytes) {
  __shared__ uint32_t warp_base[kStageBlock / 32 + 1];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  WarpScratch& ws = warp_scratch();
  uint32_t b_lo, b_hi;
  block_specs(lo, hi, b_lo, b_hi);
  const bool few = b_hi - b_lo <= 32;   // then every warp works the places out by itself
  unsigned long long bytes = 0, taken = 0;
#pragma unroll 1
  for (uint32_t base = b_lo; base < b_hi; base += kStageBlock) {
    // places of the next kStageBlock Specs
    const uint32_t own = base + (few ? lane : threadIdx.x);
    const uint32_t n_own = own < b_hi ? (uint32_t)cells_of(a.rmask[own]) : 0u;
    uint32_t inc = n_own;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
      if (lane >= (uint32_t)o) inc += t;
    }
    if (!few) {
      __syncthreads();   // the run before has been read
      ws.who[lane] = inc - n_own;   // (the sweeps' scratch is free here)
      if (lane == 31) warp_base[warp] = inc;
      __syncthreads();
      if (warp == 0) {
        const uint32_t v = warp_base[lane];
        uint32_t s = v;
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, s, o);
          if (lane >= (uint32_t)o) s += t;
        }
        warp_base[lane] = s - v;
        if (lane == 31) warp_base[32] = s;
      }
      __syncthreads();
    }
    const uint32_t here = min((uint32_t)kStageBlock, b_hi - base);
#pragma unroll 1
    for (uint32_t k = warp; k < here; k += kStageBlock / 32) {
      const uint32_t i = base + k;
      const uint32_t place = few ? __shfl_sync(0xFFFFFFFFu, inc - n_own, k) : warp_base[k >> 5] + reinterpret_cast<const WarpScratch*>(&ws - warp)[k >> 5].who[k & 31u];
      const unsigned long long fbase = first_row + taken + place;
      const uint4 fm = a.rmask[i], tm = *reinterpret_cast<const uint4*>(&a.hdrs[i]);
      const unsigned long long tbase = a.hdrs[i].row_base;
      const uint2 cl = *reinterpret_cast<const uint2*>(&a.hdrs[i].cand_off);
      const uint32_t f0 = __popc(fm.x), f1 = __popc(fm.y), f2 = __popc(fm.z), f3 = __popc(fm.w), n = f0 * f1 * f2 * f3;
      MrlRow* const to = a.rows + fbase;
      if (computed_here(a, i)) {
        // (for the statistics below)
        const uint4 rec0 = lane < cl.y ? __ldg(reinterpret_cast<const uint4*>(&a.cands[cl.x + lane])) : make_uint4(0, 0, 0, 0);
        const MrlRow* const from = row_at(a.rows, a.temp, tbase);
        const bool same = tm.x == fm.x && tm.y == fm.y && tm.z == fm.z && tm.w == fm.w;
        if (!same) {   // the grid's slot of every final slot, memory after memory
          __syncwarp();   // the Spec before has been read by every lane
#pragma unroll 1
          for (uint32_t t = lane; t < f0 + f1 + f2 + f3; t += 32) {
            uint32_t mk = fm.x, tk = tm.x, slot = t;
            if (slot >= f0) { slot -= f0; mk = fm.y; tk = tm.y; if (slot >= f1) { slot -= f1; mk = fm.z; tk = tm.z; if (slot >= f2) { slot -= f2; mk = fm.w; tk = tm.w; } } }
            ws.codes[t] = (uint8_t)(__popc(tk & below(nth_set_bit(mk, slot))) - 1);
          }
          __syncwarp();
        }
        const uint32_t t0 = __popc(tm.x), t1 = __popc(tm.y), t2 = __popc(tm.z);
#pragma unroll 1
        for (uint32_t j = lane; j < n; j += 32) {
          uint32_t toff = j;
          if (!same) {
            uint32_t j0, j1, j2, j3;
            cell_slots(j, f0, f1, f2, j0, j1, j2, j3);
            toff = ((ws.codes[f0 + f1 + f2 + j3] * t2 + ws.codes[f0 + f1 + j2]) * t1 + ws.codes[f0 + j1]) * t0 + ws.codes[j0];
          }
          uint4 r = ld_row(from + toff);
          r.w = 0;
          *reinterpret_cast<uint4*>(to + j) = r;
        }
        // statistics: 12 bytes per row, 16 per record, 16 per child of every record that fits the row's limits
        if (lane == 0) bytes += n * (12ull + 16ull * cl.y);
        #pragma unroll 1
        for (uint32_t c = lane; c < cl.y; c += 32) {
          const uint4 rec = c < 32 ? rec0 : __ldg(reinterpret_cast<const uint4*>(&a.cands[cl.x + c]));
          const uint32_t kind = (rec.x >> 16) & 0xFFu, nchild = rec.x >> 24;
          uint32_t feasible = n;
          if (kind == MRL_CK_MOVE) {
            const uint32_t ml = sel4(fm.x, fm.y, fm.z, fm.w, rec.z & 0xFFu), thr = (rec.z >> 8) & 0xFFu;
            feasible = n / (uint32_t)__popc(ml) * (uint32_t)__popc(ml >> thr);   // final cells at or above the threshold
          }
          bytes += (unsigned long long)feasible * nchild * 16ull;
        }
      } else {
        #pragma unroll 1
        for (uint32_t j = lane; j < n; j += 32) *reinterpret_cast<uint4*>(to + j) = make_uint4(0, 0, 0, 0);
      }
      __syncwarp();   // the header has been read by every lane, and the rows are there for the corner
      uint32_t corner = 0;
      if (!a.mine) corner = corner_from_rows(fm, to, lane);
      if (lane == 0) {
        *reinterpret_cast<uint4*>(&a.hdrs[i]) = fm;
        a.hdrs[i].row_base = fbase;
        if (!a.mine) a.minsat[i] = corner;
      }
    }
    taken += few ? __shfl_sync(0xFFFFFFFFu, inc, 31) : warp_base[32];
  }
  for (int o = 16; o > 0; o >>= 1) bytes += __shfl_xor_sync(0xFFFFFFFFu, bytes, o);
  if (lane == 0 && bytes) atomicAdd(block_bytes, bytes);
  return taken;
}

// Out of line: a grid-wide barrier is a hundred instructions, a stage has a dozen of them, and what a small
// stage waits for is instructions.
__device__ __noinline__ void team_barrier(uint32_t team) {
  if (team == TEAM_GRID) {
    cg::this_grid().sync();
  } else if (team == TEAM_CLUSTER) {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
  } else {
    __syncthreads();
  }
}

// A block alone reads and writes everything through its own L1, where a hit takes a tenth of the 700
// cycles that a dependent read from L2 was measured to take here, and a small plan is nothing but chains
// of such reads. So what the run touches is brought in at its start, as far as L1 reaches; stores
// update what they hit.
__device__ __noinline__ void warm_l1(const StageArgs& a) {
  const uint32_t lo = __ldg(&a.stages[a.stage_lo]).x, hi = __ldg(&a.stages[a.stage_hi - 1]).y, n = hi - lo;
  uint32_t acc = 0, left = kWarmLines;
  auto touch = [&](const void* p, size_t bytes) {
    const uint32_t lines = (uint32_t)min((size_t)left, (bytes + 127) / 128);
    #pragma unroll 1
    for (uint32_t k = threadIdx.x; k < lines; k += kStageBlock) acc ^= *reinterpret_cast<const uint32_t*>(static_cast<const char*>(p) + k * 128u);
    left -= lines;
  };
  const SpecHdr* const h = a.hdrs + lo;
  touch(h, n * sizeof(SpecHdr));
  const uint32_t c_lo = h[0].cand_off, c_hi = h[n - 1].cand_off + h[n - 1].ncand;
  touch(a.rmask + lo, n * sizeof(uint4));
  touch(a.minsat + lo, n * sizeof(uint32_t));
  touch(a.cands + c_lo, (size_t)(c_hi - c_lo) * sizeof(CandRec));
  if (acc == 0x9E3779B9u && left > kWarmLines) a.ctl->scratch[0] = acc;   // (never: the loads are to be made)
}

// A run of stages, each start to finish, by one team of blocks: the grid (cooperative launch), one
// cluster, or one block. Every thread of the team reaches every barrier: what decides the control
// flow (totals, the error word) is read from device memory after a barrier and written again only after
// a later one, so all threads take the same branches. The one exception is the sweep that last changed a
// cell (sweep_changed_a_cell).
//
// What bounds a small stage is the number of barriers: a grid-wide one takes 2 us and more, and a
// 2x2x2 Matmul search has 86 stages of 9 Specs on average. So the team fits the stage - a cluster's
// barrier takes a fraction of that and a block's next to nothing - and a stage makes as few as its
// phases depend on each other: 5 without same-stage children, 10 with them and one pass.
__global__ void __launch_bounds__(kStageBlock, 1) stage_kernel(const __grid_constant__ StageArgs a) {
  const uint32_t gtid = blockIdx.x * kStageBlock + threadIdx.x;
  const uint32_t gthreads = gridDim.x * kStageBlock;
  const uint32_t gwarp = gtid >> 5, gwarps = gthreads >> 5;
  FillCtl* const ctl = a.ctl;
  uint32_t syncs = 0;
  auto team_sync = [&]() {
    syncs++;
    team_barrier(a.team);
  };
  if (ctl->error) return;   // an earlier stage failed: the host repairs and resumes (uniform: nothing writes it before the first barrier)
  // statistics of the block: candidates evaluated and rows gathered by the unordered phase; by the
  // sweeps; items the sweeps solved cells of; bytes of the finished rows
  __shared__ unsigned long long block_stats[6], phase_ns[8];
  __shared__ StageCtl own_ctl;
  StageCtl* const sc = a.team == TEAM_BLOCK ? &own_ctl : &ctl->stage;
  if (threadIdx.x < 6) block_stats[threadIdx.x] = 0;
  if (threadIdx.x < 8) phase_ns[threadIdx.x] = 0;
  if (threadIdx.x < sizeof(StageCtl) / 4) reinterpret_cast<uint32_t*>(&own_ctl)[threadIdx.x] = 0;
  __syncthreads();
  auto get = [](const auto* p) { return *reinterpret_cast<const volatile std::remove_const_t<std::remove_pointer_t<decltype(p)>>*>(p); };   // past L1: others write it
  unsigned long long final_top = ctl->final_top;   // rows of the table; written below behind a barrier
  unsigned long long t_last = 0, st_cells = 0, st_early = 0;
  uint32_t n_sweeps = 0, n_passes = 0;
  if (gtid == 0) asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_last));
  // device time since the last mark goes to part ph (thread 0 only; after a barrier)
#define MARK(ph) do { if (gtid == 0) { unsigned long long t_now; asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_now)); \
                                       phase_ns[ph] += t_now - t_last; t_last = t_now; } } while (0)
  if (a.team == TEAM_BLOCK) warm_l1(a);
  #pragma unroll 1
  for (uint32_t st = a.stage_lo; st < a.stage_hi; st++) {
    const uint2 ids = __ldg(&a.stages[st]);
    const uint32_t lo = ids.x, hi = ids.y;
    bool failed = false;
    if (a.solve) {
      uint32_t ph = 0;   // phases that hand out items take the counters in turn; one is cleared four phases ahead
      HotArgs h;
      h.hdrs = a.hdrs; h.cands = a.cands; h.rows = a.rows; h.temp = a.temp; h.temp_cap = a.temp_cap; h.sspec = a.sspec - lo;
      h.items = a.items; h.n_items = 0; h.next_item = nullptr;
      auto hand_out = [&](uint32_t n_items) {
        h.n_items = n_items;
        h.next_item = &sc->next_item[ph & 7];
        if (gtid == 0) sc->next_item[(ph + 4) & 7] = 0;
        ph++;
      };
      auto too_small = [&](unsigned long long rows_early, unsigned long long rows_late, unsigned long long items) {
        if (rows_early <= a.temp_cap && rows_late <= a.temp_cap && items <= a.item_cap) return false;
        if (gtid == 0) {
          ctl->failed_stage = st;
          ctl->error |= MRL_ERR_WORKING;
          ctl->need_temp = max(rows_early, rows_late);
          ctl->need_items = items;
        }
        return true;
      };
      if (a.mine && st) {
        phase_minsat(a, __ldg(&a.stages[st - 1]).x, __ldg(&a.stages[st - 1]).y, gwarp, gwarps);
        team_sync();
      }
      const bool fused = a.team != TEAM_GRID;
      bool any_late;
      if (fused) {
        phase_early_fused(a, h, sc, lo, hi, gwarp, gwarps, st, block_stats);
        team_sync();
        any_late = get(&sc->any_late) == st + 1;
        MARK(MRL_PH_EARLY);
      } else {
        phase_records(a, sc, lo, hi, gwarp, gwarps, st);
        team_sync();
        any_late = get(&sc->any_late) == st + 1;
        phase_place_early(a, sc, lo, hi, gwarp, gwarps, any_late);
        team_sync();
        MARK(MRL_PH_SETUP);
      }
      const unsigned long long cells = get(&sc->rows_early);
      const uint32_t n_early_items = get(&sc->n_items_early);
      failed = too_small(cells, 0, n_early_items);
      if (!failed && cells) {
        st_cells += cells;
        st_early += cells;
        if (n_early_items) {
          hand_out(n_early_items);
          phase_early(h, block_stats);
          team_sync();
          MARK(MRL_PH_EARLY);
          hand_out(n_early_items);
          phase_real_masks<true>(h, a.rmask, false);
          team_sync();
          MARK(MRL_PH_EARLY_MASKS);
        }
        uint32_t sweep = 0;
        unsigned long long rows_before = 0;
        if (!any_late && !fused) phase_place_late(a, sc, lo, hi, gwarp, gwarps, 0);   // headers only; the places of the rows need no barrier behind it
        #pragma unroll 1
        for (uint32_t pass = 0; any_late; pass++) {
          if (pass >= (uint32_t)kMaxPasses) { failed = true; if (gtid == 0) { ctl->failed_stage = st; ctl->error |= MRL_ERR_PASSES; } break; }
          phase_place_late(a, sc, lo, hi, gwarp, gwarps, pass);
          team_sync();
          const unsigned long long rows = get(&sc->rows_late);
          const uint32_t n_items = get(&sc->n_items);
          if ((failed = too_small(0, rows, n_items))) break;
          MARK(MRL_PH_PASS_SETUP);
          if (pass) {
            hand_out(n_items);
            phase_refine(h);
            team_sync();
            MARK(MRL_PH_INIT);
          } else {
            #pragma unroll 1
            for (uint32_t i = lo + gtid; i < hi; i += gthreads)   // what the unordered phase found real has been used
              if (computed_here(a, i) && a.sspec[i - lo].n_late) a.rmask[i] = make_uint4(1u, 1u, 1u, 1u);
          }
          st_cells += rows - rows_before;
          rows_before = rows;
          const uint32_t sweep_before = sweep;
          #pragma unroll 1
          for (bool first = true;; first = false) {
            sweep++;
            uint4* const now = a.changed[sweep % 3], *const idle = a.changed[(sweep + 1) % 3];
            const uint4* const before = a.changed[(sweep + 2) % 3];
            if (sweep > 1)   // the first sweeps' are zero from phase_place_late
              #pragma unroll 1
              for (uint32_t i = gtid; i < hi - lo; i += gthreads) idle[i] = make_uint4(0, 0, 0, 0);
            hand_out(n_items);
            if (first && !pass) phase_sweep<true>(h, SWEEP_ALL, lo, before, now, sweep, &sc->any_changed, block_stats);
            else phase_sweep<false>(h, first ? SWEEP_NEW : SWEEP_CHANGED, lo, before, now, sweep, &sc->any_changed, block_stats);
            team_sync();
            MARK(first ? MRL_PH_SWEEP_FIRST : MRL_PH_SWEEP_MORE);
            if (!sweep_changed_a_cell(get(&sc->any_changed), sweep)) break;   // nothing changed anywhere: the stage's cells are consistent
            if (sweep - sweep_before >= (uint32_t)kMaxSweeps) {   // more sweeps than the limits lattice has diagonals: give up rather than spin
              failed = true;
              if (gtid == 0) { ctl->failed_stage = st; ctl->error |= MRL_ERR_PASSES; }
              break;
            }
          }
          if (failed) break;
          n_sweeps += sweep - sweep_before;
          n_passes++;
          if (pass) {
            #pragma unroll 1
            for (uint32_t i = lo + gtid; i < hi; i += gthreads)
              if (computed_here(a, i) && a.sspec[i - lo].n_late && a.sspec[i - lo].dirty) a.rmask[i] = make_uint4(1u, 1u, 1u, 1u);
            team_sync();
          }
          if (gtid == 0) sc->n_items = 0;
          hand_out(n_items);
          phase_real_masks<false>(h, a.rmask, pass != 0);
          team_sync();
          phase_check_grids(a, sc, lo, hi, gwarp, gwarps, pass);
          if (a.place && gridDim.x > 1) phase_count(a, lo, hi);   // for when no grid grows
          team_sync();
          MARK(MRL_PH_PASS_MASKS);
          if (get(&sc->grew) != pass + 1) break;   // every working grid is consistent
        }
        if (!any_late && !failed && gridDim.x > 1) {
          if (a.place) phase_count(a, lo, hi);
          team_sync();
        }
      }
    } else if (gridDim.x > 1) {
      phase_count(a, lo, hi);
      team_sync();
    }
    if (!failed && a.place) {
      unsigned long long before = 0, total = 0;
      bool fits = false;
      if (gridDim.x > 1) {
        #pragma unroll 1
        for (uint32_t b = threadIdx.x; b < gridDim.x; b += kStageBlock) {
          const unsigned long long v = get(&a.block_sums[b]);
          total += v;
          if (b < blockIdx.x) before += v;
        }
        before = block_sum(before);
        total = block_sum(total);
      } else {   // a block alone learns its total from the compaction, where no total could be too large
        fits = a.solve && final_top + get(&sc->rows_early) + get(&sc->rows_late) <= a.row_cap;
        if (!fits) {
          #pragma unroll 1
          for (uint32_t i = lo + threadIdx.x; i < hi; i += kStageBlock) total += cells_of(a.rmask[i]);
          total = block_sum(total);
        }
      }
      if (!fits && final_top + total > a.row_cap) {   // uniform
        failed = true;
        if (gtid == 0) {
          ctl->failed_stage = st;
          ctl->error |= MRL_ERR_TABLE;
          ctl->need_rows = final_top + total;
        }
      } else {
        const unsigned long long taken = phase_compact(a, lo, hi, final_top + before, &block_stats[5]);
        if (gridDim.x == 1) total = taken;
        __syncthreads();   // the counters read above are cleared below
        if (gtid == 0) {
          ctl->stage_first_row = final_top;
          ctl->stage_rows = total;
          sc->rows_early = sc->rows_late = 0;
          sc->n_items_early = sc->n_items = sc->any_changed = sc->grew = 0;
#pragma unroll
          for (int k = 0; k < 8; k++) sc->next_item[k] = 0;
        }
        final_top += total;
        if (gtid == 0) ctl->final_top = final_top;
        if (st + 1 < a.stage_hi) team_sync();
        MARK(MRL_PH_SETUP);
      }
    }
    if (failed) break;   // uniform
  }
#undef MARK
  __syncthreads();
  if (threadIdx.x == 0 && (block_stats[0] | block_stats[1] | block_stats[2] | block_stats[4] | block_stats[5])) {
    atomicAdd(&ctl->st_cands, block_stats[0] + block_stats[2]);
    atomicAdd(&ctl->st_lookups, block_stats[1] + block_stats[3]);
    atomicAdd(&ctl->st_late_cands, block_stats[2]);
    atomicAdd(&ctl->st_late_items, block_stats[4]);
    atomicAdd(&ctl->st_final_bytes, block_stats[5]);
  }
  if (gtid == 0) {
    ctl->st_sweeps += n_sweeps;
    ctl->st_passes += n_passes;
    ctl->st_cells += st_cells;
    ctl->st_early_cells += st_early;
    ctl->st_syncs += syncs;
    for (int k = 0; k < 8; k++) ctl->st_phase_ns[k] += phase_ns[k];
  }
}

// Consistency check of a finished table: at sampled (or all) points of the limits lattice, for
// sampled (or all) Specs, the direct solve from the children's tables - every candidate record,
// no re-use of neighbouring cells - must equal what the Spec's own table returns there. Every
// point where that holds is a point where the table satisfies the defining recurrence of the
// fill, whatever grid the table is stored on.
__global__ void __launch_bounds__(kBlock)
verify_points_kernel(const SpecHdr* hdrs, const CandRec* __restrict__ cands, const MrlRow* rows, uint32_t n_specs,
                     uint32_t top_pack, unsigned long long first, unsigned long long count,
                     unsigned long long total_points, unsigned long long seed, int exhaustive,
                     unsigned long long* out /* [0] mismatches, [1] first bad sample */) {
  const unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const uint32_t e0 = code_of(top_pack, 0) + 1, e1 = code_of(top_pack, 1) + 1, e2 = code_of(top_pack, 2) + 1,
                 e3 = code_of(top_pack, 3) + 1;
  const unsigned long long per_spec = (unsigned long long)e0 * e1 * e2 * e3;
  unsigned long long s = first + i;
  if (!exhaustive) {
    // splitmix64 of (seed, sample index): a point of the (Spec x lattice) product
    unsigned long long z = seed + 0x9E3779B97F4A7C15ull * (s + 1);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    s = z % total_points;
  }
  const uint32_t spec = (uint32_t)(s / per_spec);
  uint32_t p = (uint32_t)(s % per_spec);
  const uint32_t c0 = p % e0; p /= e0;
  const uint32_t c1 = p % e1; p /= e1;
  const uint32_t c2 = p % e2;
  const uint32_t c3 = p / e2;
  const uint32_t cpack = c0 | (c1 << 8) | (c2 << 16) | (c3 << 24);
  Tally tally = {0, 0};
  const Best k = solve_point(hdrs, cands, rows, rows, spec, cpack, tally);
  const uint4 r = lookup(hdrs, rows, rows, spec, below(c0), below(c1), below(c2), below(c3));
  if (k.main != r.x || k.peaks != r.y || k.tail != r.z) {
    atomicAdd(&out[0], 1ull);
    atomicMin(&out[1], first + i);
  }
}

// Point lookups for get: the row of (Spec id, packed limit codes), into a dense buffer.
__global__ void lookup_rows_kernel(const SpecHdr* hdrs, const MrlRow* rows, const uint2* __restrict__ queries,
                                   unsigned long long n, MrlRow* __restrict__ out) {
  const unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint2 q = queries[i];
  const uint4 r = lookup(hdrs, rows, rows, q.x, below(code_of(q.y, 0)), below(code_of(q.y, 1)), below(code_of(q.y, 2)),
                         below(code_of(q.y, 3)));
  *reinterpret_cast<uint4*>(out + i) = r;
}

// The same for Specs of a plan made on the device, named by family and operands: a Spec's id is the
// number of existing Specs before its position. aux = 1 in the answer: the Spec does not exist.
struct PackedQuery { unsigned long long spec; uint32_t cpack, pad; };
__global__ void __launch_bounds__(kBlock)
lookup_packed_kernel(const mrl::DpTables t, const SpecHdr* hdrs, const MrlRow* rows, const PackedQuery* queries, unsigned long long n,
                     MrlRow* out) {
  const unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const PackedQuery q = queries[i];
  const uint32_t pos = mrl::dp_pos(t, t.fams[q.spec >> 48], (uint32_t)(q.spec >> 32) & 0xFFFFu, (uint32_t)(q.spec >> 16) & 0xFFFFu,
                                   (uint32_t)q.spec & 0xFFFFu);
  uint4 r = make_uint4(MRL_UNSAT, MRL_UNSAT, MRL_UNSAT, 1u);
  if ((t.rank[pos >> 5].x >> (pos & 31u)) & 1u) {
    r = lookup(hdrs, rows, rows, mrl::dp_id(t, pos), below(code_of(q.cpack, 0)), below(code_of(q.cpack, 1)), below(code_of(q.cpack, 2)),
               below(code_of(q.cpack, 3)));
    r.w = 0;
  }
  *reinterpret_cast<uint4*>(out + i) = r;
}

// The implementation tree of one Spec: from its row, the record with the stored action, that record's
// sub-Specs at the limits the action leaves them, and so on, level by level; a node per warp, its
// records over the lanes. The host turns the nodes into text. One block: a tree has tens of nodes, and a
// level costs four dependent reads.
constexpr uint32_t kWalkMost = 2048;
__global__ void __launch_bounds__(kBlock)
walk_kernel(const mrl::DpTables t, const unsigned long long* desc, const SpecHdr* hdrs, const CandRec* __restrict__ cands, const MrlRow* rows,
            uint32_t n_specs, unsigned long long root, uint32_t root_is_packed, uint32_t cpack, mrl::WalkNode* nodes, uint32_t* count) {
  __shared__ uint32_t n, level_end;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    mrl::WalkNode r;
    memset(&r, 0, sizeof(r));
    r.cpack = cpack;
    r.id = (uint32_t)root;
    if (root_is_packed) {
      const uint32_t pos = mrl::dp_pos(t, t.fams[root >> 48], (uint32_t)(root >> 32) & 0xFFFFu, (uint32_t)(root >> 16) & 0xFFFFu, (uint32_t)root & 0xFFFFu);
      r.id = (t.rank[pos >> 5].x >> (pos & 31u)) & 1u ? mrl::dp_id(t, pos) : 0xFFFFFFFFu;
    }
    nodes[0] = r;
    n = level_end = 1;
  }
  __syncthreads();
  uint32_t lo = 0;
  for (uint32_t depth = 0; depth < 512 && lo < level_end; depth++) {
    const uint32_t hi = level_end;
    for (uint32_t k = lo + warp; k < hi; k += kBlock / 32) {
      const uint32_t id = nodes[k].id, cp = nodes[k].cpack;
      if (id >= n_specs) { if (lane == 0) nodes[k].status = mrl::WALK_NO_SPEC; continue; }
      const uint4 r = lookup(hdrs, rows, rows, id, below(code_of(cp, 0)), below(code_of(cp, 1)), below(code_of(cp, 2)), below(code_of(cp, 3)));
      if (lane == 0) {
        nodes[k].spec = desc ? desc[id] : 0ull;
        nodes[k].main = r.x; nodes[k].peaks = r.y; nodes[k].tail = r.z;
      }
      if (r.z == MRL_UNSAT) { if (lane == 0) nodes[k].status = mrl::WALK_UNSAT; continue; }
      const uint2 cl = *reinterpret_cast<const uint2*>(&hdrs[id].cand_off);
      bool found = false;
      for (uint32_t c0 = 0; c0 < cl.y && !found; c0 += 32) {
        const uint32_t c = c0 + lane;
        const uint32_t head = c < cl.y ? __ldg(reinterpret_cast<const uint32_t*>(&cands[cl.x + c])) : 0u;
        const bool hit = c < cl.y && (head & 0xFFFFu) == (r.z & 0xFFFFu);
        found = __any_sync(0xFFFFFFFFu, hit);
        if (!hit) continue;
        const CandRec rec = cands[cl.x + c];
        uint32_t child_cp = cp;
        if (rec.kind == MRL_CK_MOVE) {
          const uint32_t lv = code_of(cp, rec.level), q = lv >= rec.thr_code ? child_code(rec.level, lv, rec.units) : 0u;
          child_cp = (cp & ~(0xFFu << (8 * rec.level))) | (q << (8 * rec.level));
          if (lv < rec.thr_code) nodes[k].status = mrl::WALK_BAD;
        }
        const uint32_t at = atomicAdd(&n, (uint32_t)rec.nchild);
        nodes[k].first_child = at;
        nodes[k].n_child = rec.nchild;
        for (uint32_t j = 0; j < rec.nchild; j++)
          if (at + j < kWalkMost) {
            mrl::WalkNode q;
            memset(&q, 0, sizeof(q));
            q.id = rec.child[j];
            q.cpack = child_cp;
            nodes[at + j] = q;
          }
      }
      if (!found && lane == 0) nodes[k].status = mrl::WALK_BAD;
    }
    __syncthreads();
    if (threadIdx.x == 0) level_end = min(n, kWalkMost);
    lo = hi;
    __syncthreads();
  }
  if (threadIdx.x == 0) *count = n;
}

// The finished table's headers as the two arrays a bulk export hands out.
__global__ void __launch_bounds__(kBlock) export_headers_kernel(const SpecHdr* hdrs, uint32_t n_specs, uint4* masks, unsigned long long* first_row) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_specs) return;
  masks[i] = *reinterpret_cast<const uint4*>(&hdrs[i]);
  first_row[i] = hdrs[i].row_base;
}

__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// Sum over all Specs of a hash of (id, masks, rows in cell order). The sum commutes, and where a
// Spec's rows lie in the table does not enter, so two fills of one plan agree however their
// tables are laid out.
__global__ void __launch_bounds__(kBlock)
checksum_kernel(const SpecHdr* hdrs, const MrlRow* rows, uint32_t n_specs, unsigned long long* out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long h = 0;
  if (i < n_specs) {
    const uint4 m = *reinterpret_cast<const uint4*>(&hdrs[i]);
    const unsigned long long base = hdrs[i].row_base;
    const unsigned long long n = (unsigned long long)__popc(m.x) * __popc(m.y) * __popc(m.z) * __popc(m.w);
    h = mix64(0x9E3779B97F4A7C15ull * (i + 1ull));
    h = mix64(h ^ (((unsigned long long)m.x << 32) | m.y));
    h = mix64(h ^ (((unsigned long long)m.z << 32) | m.w));
    for (unsigned long long j = 0; j < n; j++) {
      const uint4 r = *reinterpret_cast<const uint4*>(rows + base + j);
      h = mix64(h ^ (((unsigned long long)r.x << 32) | r.y));
      h = mix64(h ^ r.z);
    }
  }
  for (int o = 16; o > 0; o >>= 1) h += __shfl_xor_sync(0xFFFFFFFFu, h, o);
  if ((threadIdx.x & 31) == 0 && h) atomicAdd(out, h);
}

// Candidate records that arrived on the device without passing through this host's planner:
// every field a kernel indexes with must be in range.
__global__ void __launch_bounds__(kBlock)
check_records_kernel(const SpecHdr* hdrs, const CandRec* __restrict__ cands, uint32_t n_specs, unsigned long long n_cands,
                     uint32_t* error) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_specs) return;
  const uint2 cl = *reinterpret_cast<const uint2*>(&hdrs[i].cand_off);
  bool bad = (unsigned long long)cl.x + cl.y > n_cands;
  for (uint32_t ci = 0; ci < cl.y && !bad; ci++) {
    const CandRec c = cands[cl.x + ci];
    bad = c.kind > MRL_CK_BLOCK || c.nchild > 3 || c.level > 3 || c.thr_code > 30 || c.peak_code > 31 || c.late > 1 ||
          (c.kind == MRL_CK_LEAF) != (c.nchild == 0);
    for (uint32_t j = 0; j < c.nchild && !bad; j++) bad = c.child[j] >= n_specs;
  }
  if (bad) atomicOr(error, (uint32_t)MRL_ERR_CHILD);
}

}  // namespace

namespace mrl {

#define CK(x)                                                                              \
  do {                                                                                     \
    cudaError_t e_ = (x);                                                                  \
    if (e_ != cudaSuccess) {                                                               \
      snprintf(err_, sizeof(err_), "%s failed: %s", #x, cudaGetErrorString(e_));           \
      return -1;                                                                           \
    }                                                                                      \
  } while (0)

constexpr size_t kStageSmem = (kStageBlock / 32) * sizeof(WarpScratch);

static size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

// The team for a stage of n Specs of one kind, log-shape sum and level rank. A grid-wide barrier takes
// 2 us and a stage has 5 to 20 of them, a cluster's a fraction of that, a block's less still; against
// that stands the work, and Specs differ in it by orders of magnitude: their grids grow with the
// operands' volume, and with how many of the operands are still in the slowest memory (the finished
// rows of a Matmul stage: 2 per Spec at 1x1x2, 200 at 2x8x4, 1 900 at 8x8x8 with all operands there, a
// tenth of that with all in the others).
constexpr uint32_t kMergeSpecs = 1u << 18;
constexpr uint32_t kBlockSpecs = 24, kBlockWork = 3000, kClusterSpecs = 256, kClusterWork = 20000;
static uint32_t team_of_stage(uint32_t n, uint32_t kind, uint32_t shape_sum, uint32_t level_rank) {
  const int below_top = (kind == K_MOVE || kind == K_FILL_ZERO ? (int)GL : 3 * (int)GL) - (int)level_rank;
  const uint32_t shift = shape_sum + (uint32_t)std::min(3, std::max(0, 4 - below_top));
  const uint64_t work = shift < 32 ? (uint64_t)n << shift : ~uint64_t(0);
  if (n <= kBlockSpecs && work <= kBlockWork) return TEAM_BLOCK;
  return n <= kClusterSpecs && work <= kClusterWork ? TEAM_CLUSTER : TEAM_GRID;
}

struct DeviceFill::DevTables {
  DpTables t;
};

DeviceFill::DeviceFill() {}
DeviceFill::~DeviceFill() { release(); }

int DeviceFill::too_large_() {
  snprintf(err_, sizeof(err_),
           "this fill needs more than the %zu bytes of device memory the no-allocation entry point has; "
           "use mrl_top_down_many for it", buf_bytes_);
  return -5;
}

int DeviceFill::alloc_(void** p, size_t bytes) {
  bytes = std::max<size_t>(bytes, 256);
  if (fixed_) {
    const size_t off = align256(buf_off_);
    if (off + bytes > buf_bytes_) return too_large_();
    *p = buf_ + off;
    buf_off_ = off + bytes;
    return 0;
  }
  cudaError_t e = cudaMalloc(p, bytes);
  if (e != cudaSuccess) {
    cudaGetLastError();
    snprintf(err_, sizeof(err_), "out of device memory: cudaMalloc of %zu bytes failed (%s)", bytes, cudaGetErrorString(e));
    return -6;
  }
  return 0;
}

void DeviceFill::drop_(DevBuf& b) {
  if (b.p && !fixed_) cudaFree(b.p);
  b.p = nullptr;
  b.cap = 0;
}

// A cudaMalloc or cudaFree costs 50 us to milliseconds (seconds, in the tail) against the 1 to 60
// ms of a small fill, and a plan has some twenty buffers, so buffers stay from plan to plan. What
// a large plan leaves behind is given back when the next plan needs less than a quarter of it (a fill that
// had to enlarge a buffer keeps it for the next one of its size, which asks for the first size again).
bool DeviceFill::oversized_(const DevBuf& b, size_t bytes) { return b.cap > (size_t(256) << 20) && b.cap / 4 > bytes; }
int DeviceFill::reserve_(DevBuf& b, size_t bytes, bool give_back) {
  bytes = std::max<size_t>(bytes, 256);
  if (!fixed_ && b.cap >= bytes && !(give_back && oversized_(b, bytes))) return 0;
  if (!fixed_ && b.p) {
    CK(cudaStreamSynchronize(stream_));
    drop_(b);
  }
  const size_t want = fixed_ ? bytes : (bytes < (size_t(64) << 20) ? bytes + bytes / 4 : bytes);
  int rc = alloc_(&b.p, want);
  if (rc) { b.p = nullptr; b.cap = 0; return rc; }
  b.cap = want;
  return 0;
}

int DeviceFill::reserve_host_(size_t bytes) {
  if (h_stage_bytes_ >= bytes) return 0;
  if (fixed_) {   // pinning memory is an allocation the no-allocation entry point does not make
    h_pageable_.resize(bytes);
    h_stage_ = h_pageable_.data();
    h_stage_bytes_ = bytes;
    return 0;
  }
  if (h_stage_) cudaFreeHost(h_stage_);
  h_stage_ = nullptr;
  h_stage_bytes_ = 0;
  const size_t want = std::max<size_t>(bytes + std::min<size_t>(bytes / 2, size_t(1) << 20), size_t(64) << 10);
  CK(cudaHostAlloc(&h_stage_, want, cudaHostAllocDefault));
  h_stage_bytes_ = want;
  return 0;
}

int DeviceFill::drop_all_() {
  begin_plan_();
  CK(cudaStreamSynchronize(stream_));
  for (DevBuf* b : {&b_ctl_, &b_hdrs_, &b_cands_, &b_spec_, &b_stage_specs_, &b_mine_, &b_stages_, &b_items_, &b_temp_, &b_rows_,
                    &b_lookup_, &b_tables_, &b_bits_, &b_rank_, &b_desc_, &b_stage_lo_})
    drop_(*b);
  return 0;
}

void DeviceFill::release() {
  wait_upload();
  for (DevBuf* b : {&b_ctl_, &b_hdrs_, &b_cands_, &b_spec_, &b_stage_specs_, &b_mine_, &b_stages_, &b_items_, &b_temp_, &b_rows_,
                    &b_lookup_, &b_tables_, &b_bits_, &b_rank_, &b_desc_, &b_stage_lo_})
    drop_(*b);
  tab_.reset();
  buf_off_ = 0;
  cands_present_ = false;
  if (h_stage_ && !fixed_) cudaFreeHost(h_stage_);
  h_stage_ = nullptr;
  h_stage_bytes_ = 0;
  if (h_ctl_ && h_ctl_ != &ctl_pageable_) cudaFreeHost(h_ctl_);
  h_ctl_ = nullptr;
  if (ev0_) cudaEventDestroy(ev0_);
  if (ev1_) cudaEventDestroy(ev1_);
  ev0_ = ev1_ = nullptr;
  if (own_stream_ && stream_) cudaStreamDestroy(stream_);
  stream_ = nullptr;
  own_stream_ = false;
}

int DeviceFill::init(int device) {
  device_ = device;
  CK(cudaSetDevice(device));
  if (!stream_) {
    CK(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking));
    own_stream_ = true;
  }
  return init_events();
}

int DeviceFill::init_events() {
  if (!ev0_) CK(cudaEventCreate(&ev0_));
  if (!ev1_) CK(cudaEventCreate(&ev1_));
  int coop = 0, per_sm = 0;
  CK(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device_));
  CK(cudaDeviceGetAttribute(&n_sm_, cudaDevAttrMultiProcessorCount, device_));
  if (!coop) { snprintf(err_, sizeof(err_), "the device does not support cooperative launches"); return -1; }
  CK(cudaFuncSetAttribute(stage_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kStageSmem));
  CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, stage_kernel, kStageBlock, kStageSmem));
  if (per_sm < 1) { snprintf(err_, sizeof(err_), "the stage kernel does not fit an SM"); return -1; }
  coop_blocks_ = per_sm * n_sm_;
  plan_blocks_ = plan_kernel_blocks_per_sm();
  if (plan_blocks_ < 1) { snprintf(err_, sizeof(err_), "the plan kernel does not fit an SM"); return -1; }
  return 0;
}

void DeviceFill::attach_buffer(void* base, size_t bytes, cudaStream_t stream, int device) {
  fixed_ = true;
  buf_ = static_cast<unsigned char*>(base);
  buf_bytes_ = bytes;
  buf_off_ = 0;
  stream_ = stream;
  own_stream_ = false;
  device_ = device;
}

int DeviceFill::set_stream(cudaStream_t s) {
  if (own_stream_ && stream_) cudaStreamDestroy(stream_);
  stream_ = s;
  own_stream_ = false;
  return 0;
}

int DeviceFill::wait_cands_(uint64_t upto_bytes) {
  if (up_threads_.empty()) return 0;
  const size_t need = std::min<uint64_t>(up_pieces_, (upto_bytes + up_piece_bytes_ - 1) / up_piece_bytes_);
  while (up_ready_ < need) {
    if (up_done_[up_ready_].load(std::memory_order_acquire)) up_ready_++;
    else if (up_err_.load(std::memory_order_relaxed) != 0) break;
    else std::this_thread::sleep_for(std::chrono::microseconds(50));
  }
  const int e = up_err_.load();
  if (up_ready_ == up_pieces_ || e != 0) {
    for (auto& th : up_threads_) th.join();
    up_threads_.clear();
  }
  if (e != 0) {
    snprintf(err_, sizeof(err_), "candidate upload failed: %s", cudaGetErrorString((cudaError_t)e));
    return -1;
  }
  return 0;
}

int DeviceFill::wait_upload() { return wait_cands_(~uint64_t(0) >> 1); }

// Forgets the plan the device holds.
void DeviceFill::begin_plan_() {
  wait_upload();   // of an earlier plan
  if (fixed_) {    // carved afresh by every plan
    for (DevBuf* b : {&b_ctl_, &b_hdrs_, &b_cands_, &b_spec_, &b_stage_specs_, &b_mine_, &b_stages_, &b_items_, &b_temp_, &b_rows_,
                      &b_lookup_, &b_tables_, &b_bits_, &b_rank_, &b_desc_, &b_stage_lo_})
      drop_(*b);
    buf_off_ = 0;
  }
  tab_.reset();
  cands_present_ = false;
  stages_.clear();
  n_specs_ = 0;
  max_stage_ = 1;
  n_cand_bytes_ = 0;
}

// Buffers a fill works in, for n_specs_ Specs in stages_ (of which a rank of `world` computes its share).
int DeviceFill::working_buffers_(bool with_mine, uint32_t world) {
  int rc;
  max_stage_ = 1;
  for (const StageIds& st : stages_) max_stage_ = std::max(max_stage_, st.hi - st.lo);
  const size_t n = std::max<uint32_t>(n_specs_, 1), ms = max_stage_;
  // per Spec: real-breakpoint masks, corner; per Spec of a stage: what the stage kernel keeps, and three
  // sweeps' changes
  const size_t o_minsat = align256(n * sizeof(uint4));
  if ((rc = reserve_(b_spec_, o_minsat + n * sizeof(uint32_t)))) return rc;
  unsigned char* p = static_cast<unsigned char*>(b_spec_.p);
  d_rmask_ = reinterpret_cast<uint4*>(p);
  d_minsat_ = reinterpret_cast<uint32_t*>(p + o_minsat);
  const size_t o_changed = align256(ms * sizeof(StageSpec)), o_sums = o_changed + 3 * align256(ms * sizeof(uint4));
  if ((rc = reserve_(b_stage_specs_, o_sums + (size_t)coop_blocks_ * sizeof(unsigned long long)))) return rc;
  p = static_cast<unsigned char*>(b_stage_specs_.p);
  d_sspec_ = p;
  for (int k = 0; k < 3; k++) d_changed_[k] = reinterpret_cast<uint4*>(p + o_changed + k * align256(ms * sizeof(uint4)));
  d_block_sums_ = reinterpret_cast<unsigned long long*>(p + o_sums);
  std::vector<uint2> ids(stages_.size());
  for (size_t k = 0; k < ids.size(); k++) ids[k] = make_uint2(stages_[k].lo, stages_[k].hi);
  if ((rc = reserve_(b_stages_, ids.size() * sizeof(uint2)))) return rc;
  if (!ids.empty()) CK(cudaMemcpyAsync(b_stages_.p, ids.data(), ids.size() * sizeof(uint2), cudaMemcpyHostToDevice, stream_));
  d_mine_ = nullptr;
  if (with_mine) {
    if ((rc = reserve_(b_mine_, n))) return rc;
    d_mine_ = static_cast<uint8_t*>(b_mine_.p);
  } else {
    drop_(b_mine_);
  }
  if (fixed_) {
    // Everything left is split once: lookup staging, work items, working rows and final rows.
    if ((rc = reserve_(b_lookup_, 64 << 10))) return rc;
    const size_t left = buf_bytes_ > align256(buf_off_) + 2048 ? buf_bytes_ - align256(buf_off_) - 2048 : 0;
    // per working cell: two rows of 16 bytes (the cell and what the unordered phase found for it),
    // under 1 byte of work items; the rest is the table
    item_cap_ = left / 64 / sizeof(WorkItem);
    temp_cap_ = left * 10 / 32 / (2 * sizeof(MrlRow));
    row_cap_ = (left - left / 64 - left * 10 / 32) / sizeof(MrlRow);
    if (item_cap_ < temp_cap_ / 32 + max_stage_ + 1) return too_large_();
    if (row_cap_ == 0) return too_large_();
    h_ctl_ = &ctl_pageable_;
  } else {
    // Starting sizes from what fills of this kind ended with (about 45 table rows per Spec; 1000
    // working cells per Spec of the largest stage, of which a rank of a sharded fill sees its
    // share), each within a part of the free memory. The table gets the largest
    // part: enlarging it later needs the old and the new copy at once. A stage that needs more than
    // these reports what it needs and is run again with larger buffers.
    const uint64_t shard = std::max<uint32_t>(1, world);
    const uint64_t stage_part = ((uint64_t)max_stage_ * 3 / 2 + shard - 1) / shard;   // Specs of the largest stage a rank solves, with slack
    uint64_t temp = std::max<uint64_t>(1u << 20, stage_part * 1000), rows = std::max<uint64_t>(1u << 20, (uint64_t)n_specs_ * 48);
    if (small_start_) temp = rows = 512;
    else if (temp * 2 * sizeof(MrlRow) > b_temp_.cap || rows * sizeof(MrlRow) > b_rows_.cap) {
      size_t free_b = 0, total_b = 0;
      CK(cudaMemGetInfo(&free_b, &total_b));
      free_b += b_temp_.cap + b_rows_.cap;
      temp = std::max<uint64_t>(1u << 20, std::min<uint64_t>(temp, free_b / 4 / (2 * sizeof(MrlRow))));
      rows = std::max<uint64_t>(1u << 20, std::min<uint64_t>(rows, free_b / 2 / sizeof(MrlRow)));
    }
    if ((rc = reserve_(b_temp_, temp * 2 * sizeof(MrlRow))) || (rc = reserve_(b_rows_, rows * sizeof(MrlRow)))) return rc;
    temp_cap_ = b_temp_.cap / (2 * sizeof(MrlRow));
    row_cap_ = b_rows_.cap / sizeof(MrlRow);
    item_cap_ = temp_cap_ / 32 + max_stage_ + 1;   // a work item holds at least 32 cells, and every Spec at most one partial item
    if (!h_ctl_) CK(cudaHostAlloc((void**)&h_ctl_, sizeof(FillCtl), cudaHostAllocDefault));
  }
  if ((rc = reserve_(b_items_, item_cap_ * sizeof(WorkItem)))) return rc;
  if (fixed_) {
    if ((rc = reserve_(b_temp_, temp_cap_ * 2 * sizeof(MrlRow)))) return rc;   // the cells, then what the unordered phase found for them
    if ((rc = reserve_(b_rows_, row_cap_ * sizeof(MrlRow)))) return rc;
  }
  d_items_ = static_cast<WorkItem*>(b_items_.p);
  d_temp_ = static_cast<MrlRow*>(b_temp_.p);
  d_rows_ = static_cast<MrlRow*>(b_rows_.p);
  return 0;
}

int DeviceFill::upload(const Plan& plan, bool skip_cands) {
  CK(cudaSetDevice(device_));
  int rc = upload_(plan, skip_cands);
  if (rc == -6) {   // what earlier plans left may be in the way
    if (drop_all_() != 0) return -1;
    rc = upload_(plan, skip_cands);
  }
  return rc;
}

int DeviceFill::upload_(const Plan& plan, bool skip_cands) {
  begin_plan_();
  if (!fixed_) for (DevBuf* b : {&b_tables_, &b_bits_, &b_rank_, &b_desc_, &b_stage_lo_}) drop_(*b);   // of plans made on the device
  n_specs_ = (uint32_t)plan.hdrs.size();
  top_pack_ = plan.top_pack();
  n_goals_ = plan.stats.n_goal_specs;
  for (const Stage& st : plan.stages) {
    StageIds s = {st.spec_lo, st.spec_hi, 0, team_of_stage(st.spec_hi - st.spec_lo, st.phase, st.shape_sum, st.level_rank)};
    if (st.spec_hi > st.spec_lo) s.cand_end = (uint64_t)plan.hdrs[st.spec_hi - 1].cand_off + plan.hdrs[st.spec_hi - 1].ncand;
    stages_.push_back(s);
  }
  int rc;
  if ((rc = reserve_(b_ctl_, 512))) return rc;
  if ((rc = reserve_(b_hdrs_, plan.hdrs.size() * sizeof(SpecHdr)))) return rc;
  if ((rc = reserve_(b_cands_, plan.cands.size() * sizeof(CandRec)))) return rc;
  d_ctl_ = static_cast<FillCtl*>(b_ctl_.p);
  d_hdrs_ = static_cast<SpecHdr*>(b_hdrs_.p);
  d_cands_ = static_cast<CandRec*>(b_cands_.p);
  if ((rc = working_buffers_(!plan.mine.empty(), plan.world))) return rc;
  h2d_bytes_ = plan.hdrs.size() * sizeof(SpecHdr) + (skip_cands ? 0 : plan.cands.size() * sizeof(CandRec)) + plan.mine.size();
  CK(cudaMemsetAsync(d_ctl_, 0, 512, stream_));
  if (!plan.hdrs.empty())
    CK(cudaMemcpyAsync(d_hdrs_, plan.hdrs.data(), plan.hdrs.size() * sizeof(SpecHdr), cudaMemcpyHostToDevice, stream_));
  n_cand_bytes_ = plan.cands.size() * sizeof(CandRec);
  if (skip_cands) {
    if (n_cand_bytes_) CK(cudaMemsetAsync(d_cands_, 0, n_cand_bytes_, stream_));   // defined until the caller's records arrive
  } else {
    cands_present_ = true;
    if (!plan.cands.empty()) {
      // The candidate records are gigabytes of pageable memory and one host thread stages about
      // 11 GB/s, so four threads copy them on their own streams, piece by piece in id order, and
      // go on after this call has returned (wait_cands_).
      const size_t total = n_cand_bytes_;
      if (fixed_ || (total < (size_t(1) << 30) && !small_start_)) {
        CK(cudaMemcpyAsync(d_cands_, plan.cands.data(), total, cudaMemcpyHostToDevice, stream_));
      } else {
        up_piece_bytes_ = small_start_ ? size_t(64) << 10 : size_t(128) << 20;
        up_pieces_ = (total + up_piece_bytes_ - 1) / up_piece_bytes_;
        up_done_.reset(new std::atomic<uint8_t>[up_pieces_]);
        for (size_t k = 0; k < up_pieces_; k++) up_done_[k].store(0, std::memory_order_relaxed);
        up_next_ = 0;
        up_err_ = 0;
        up_ready_ = 0;
        const unsigned char* src = reinterpret_cast<const unsigned char*>(plan.cands.data());
        unsigned char* dst = reinterpret_cast<unsigned char*>(d_cands_);
        for (int t = 0; t < 4; t++)
          up_threads_.emplace_back([this, src, dst, total]() {
            // Each thread stages through two small pinned buffers of its own: the copy into them
            // is a plain memcpy outside the driver, and the transfer out of them is asynchronous,
            // so the thread that launches the fill's kernels is not held up behind driver-side
            // staging of pageable memory.
            const size_t sub = size_t(8) << 20;
            unsigned char* pin[2] = {nullptr, nullptr};
            cudaEvent_t ev[2] = {nullptr, nullptr};
            bool used[2] = {false, false};
            cudaError_t e = cudaSetDevice(device_);
            cudaStream_t st = nullptr;
            if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
            for (int b = 0; b < 2 && e == cudaSuccess; b++) {
              e = cudaHostAlloc((void**)&pin[b], sub, cudaHostAllocDefault);
              if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ev[b], cudaEventDisableTiming);
            }
            unsigned turn = 0;
            while (e == cudaSuccess && up_err_.load(std::memory_order_relaxed) == 0) {
              const size_t k = up_next_.fetch_add(1);
              if (k >= up_pieces_) break;
              const size_t lo = k * up_piece_bytes_, hi = std::min(total, lo + up_piece_bytes_);
              for (size_t off = lo; off < hi && e == cudaSuccess; off += sub, turn++) {
                const int b = turn & 1;
                const size_t len = std::min(sub, hi - off);
                if (used[b]) e = cudaEventSynchronize(ev[b]);   // the buffer's last transfer is done
                if (e != cudaSuccess) break;
                memcpy(pin[b], src + off, len);
                e = cudaMemcpyAsync(dst + off, pin[b], len, cudaMemcpyHostToDevice, st);
                if (e == cudaSuccess) e = cudaEventRecord(ev[b], st);
                used[b] = true;
              }
              if (e == cudaSuccess) e = cudaStreamSynchronize(st);
              if (e == cudaSuccess) up_done_[k].store(1, std::memory_order_release);
            }
            if (st) { cudaStreamSynchronize(st); cudaStreamDestroy(st); }
            for (int b = 0; b < 2; b++) {
              if (ev[b]) cudaEventDestroy(ev[b]);
              if (pin[b]) cudaFreeHost(pin[b]);
            }
            if (e != cudaSuccess) {
              int expect = 0;
              up_err_.compare_exchange_strong(expect, (int)e);
            }
          });
      }
    }
  }
  if (d_mine_) CK(cudaMemcpyAsync(d_mine_, plan.mine.data(), plan.mine.size(), cudaMemcpyHostToDevice, stream_));
  CK(cudaStreamSynchronize(stream_));
  stats_ = FillStats();
  return 0;
}

int DeviceFill::plan(const OpTables& tab) {
  CK(cudaSetDevice(device_));
  int rc = plan_(tab);
  if (rc == -6) {   // what earlier plans left may be in the way
    if (drop_all_() != 0) return -1;
    rc = plan_(tab);
  }
  if (rc == -6) {   // no room for the planning buffers: the host planner needs none of them
    if (drop_all_() != 0) return -1;
    rc = 1;
  }
  return rc;
}

int DeviceFill::plan_(const OpTables& tab) {
  if (tab.max_records > DP_MAX_RECORDS || tab.n_positions == 0) return 1;
  begin_plan_();
  int rc;
  // tables, in one copy
  struct Part { const void* src; size_t bytes, off; };
  Part parts[] = {{tab.shapes.data(), tab.shapes.size() * sizeof(DpShape), 0},   {tab.ops.data(), tab.ops.size() * sizeof(DpOp), 0},
                  {tab.moves.data(), tab.moves.size() * sizeof(DpMove), 0},      {tab.tiles.data(), tab.tiles.size() * sizeof(u32), 0},
                  {tab.fams.data(), tab.fams.size() * sizeof(DpFam), 0},         {tab.fam_child.data(), tab.fam_child.size() * sizeof(u16), 0},
                  {tab.stage_base.data(), tab.stage_base.size() * sizeof(u32), 0},
                  {tab.products.data(), tab.products.size() * sizeof(DpProduct), 0}, {tab.lists.data(), tab.lists.size() * sizeof(u16), 0},
                  {tab.seeds.data(), tab.seeds.size() * sizeof(u64), 0}};
  size_t bytes = 0;
  for (Part& q : parts) { q.off = bytes; bytes += align256(q.bytes); }
  const u32 n_words = (tab.n_positions + 31) / 32, n_stages = (u32)tab.stage_base.size();
  const size_t back = align256(sizeof(PlanCtl)) + align256((n_stages + 1) * sizeof(u32));   // what comes back
  if ((rc = reserve_host_(std::max(bytes, back)))) return rc;
  for (const Part& q : parts) if (q.bytes) memcpy(static_cast<unsigned char*>(h_stage_) + q.off, q.src, q.bytes);
  const size_t word_bytes = align256((size_t)n_words * sizeof(u32));
  // The closure's queue has room for every position (8 bytes each: 63 MB at size 8 in one dtype), and lies in
  // the working rows, which are far larger and idle until the fill; a fixed buffer carves those last.
  const size_t queue_bytes = (size_t)tab.n_positions * sizeof(u64);
  if (!fixed_ && (rc = reserve_(b_temp_, queue_bytes, false))) return rc;
  if ((rc = reserve_(b_ctl_, 512)) || (rc = reserve_(b_tables_, bytes)) || (rc = reserve_(b_bits_, word_bytes + (fixed_ ? queue_bytes : 0))) ||
      (rc = reserve_(b_rank_, (size_t)n_words * sizeof(uint2))) || (rc = reserve_(b_stage_lo_, back + (size_t)plan_blocks_ * n_sm_ * sizeof(unsigned long long))))
    return rc == -5 ? 1 : rc;
  d_ctl_ = static_cast<FillCtl*>(b_ctl_.p);
  CK(cudaMemcpyAsync(b_tables_.p, h_stage_, bytes, cudaMemcpyHostToDevice, stream_));
  CK(cudaMemsetAsync(b_bits_.p, 0, word_bytes, stream_));
  CK(cudaMemsetAsync(b_stage_lo_.p, 0, sizeof(PlanCtl), stream_));
  PlanArgs a;
  memset(&a, 0, sizeof(a));
  const unsigned char* const base = static_cast<unsigned char*>(b_tables_.p);
  a.t.shapes = reinterpret_cast<const DpShape*>(base + parts[0].off);
  a.t.ops = reinterpret_cast<const DpOp*>(base + parts[1].off);
  a.t.moves = reinterpret_cast<const DpMove*>(base + parts[2].off);
  a.t.tiles = reinterpret_cast<const u32*>(base + parts[3].off);
  a.t.fams = reinterpret_cast<const DpFam*>(base + parts[4].off);
  a.t.fam_child = reinterpret_cast<const u16*>(base + parts[5].off);
  a.stage_base = reinterpret_cast<const u32*>(base + parts[6].off);
  a.products = reinterpret_cast<const DpProduct*>(base + parts[7].off);
  a.lists = reinterpret_cast<const u16*>(base + parts[8].off);
  a.seeds = reinterpret_cast<const u64*>(base + parts[9].off);
  a.n_stages = n_stages;
  a.n_products = (u32)tab.products.size();
  a.n_seeds = (u32)tab.seeds.size();
  a.n_words = n_words;
  a.found = static_cast<u32*>(b_bits_.p);
  a.queue = fixed_ ? reinterpret_cast<u64*>(static_cast<unsigned char*>(b_bits_.p) + word_bytes) : static_cast<u64*>(b_temp_.p);
  a.rank = static_cast<uint2*>(b_rank_.p);
  a.t.rank = a.rank;
  unsigned char* const res = static_cast<unsigned char*>(b_stage_lo_.p);
  a.ctl = reinterpret_cast<PlanCtl*>(res);
  a.stage_lo = reinterpret_cast<u32*>(res + align256(sizeof(PlanCtl)));
  a.block_sums = reinterpret_cast<unsigned long long*>(res + back);
  const PlanCtl* const ctl = static_cast<const PlanCtl*>(h_stage_);
  const u32* const lo = reinterpret_cast<const u32*>(static_cast<unsigned char*>(h_stage_) + align256(sizeof(PlanCtl)));
  // A warp per Spec: the grid follows the positions, up to what is co-resident. While positions are
  // few, headers and records for all of them are reserved ahead and one launch does everything;
  // otherwise the sizes come back after the closure, and again after the records are counted.
  const u32 max_blocks = (u32)(plan_blocks_ * n_sm_);
  auto blocks = [&](uint64_t specs) { return (int)std::min<uint64_t>(max_blocks, std::max<uint64_t>(8, (specs + 7) / 8)); };
  uint64_t want_specs = 0, want_cands = 0;
  if (!fixed_) {
    const uint64_t most = (uint64_t)tab.n_positions * tab.max_records;
    want_specs = std::min<uint64_t>(tab.n_positions, 1u << 16);
    want_cands = std::min<uint64_t>(most, 1u << 17);
  }
  int phases = fixed_ ? DPP_CLOSURE : DPP_CLOSURE | DPP_SPECS | DPP_RECORDS;
  for (int attempt = 0;; attempt++) {
    if (phases & DPP_SPECS) {
      if ((rc = reserve_(b_hdrs_, want_specs * sizeof(SpecHdr), false)) || (rc = reserve_(b_desc_, want_specs * sizeof(u64), false)))
        return rc == -5 ? 1 : rc;
      if ((phases & DPP_RECORDS) && (rc = reserve_(b_cands_, want_cands * sizeof(CandRec), false))) return rc == -5 ? 1 : rc;
    }
    a.hdrs = static_cast<SpecHdr*>(b_hdrs_.p);
    a.desc = static_cast<u64*>(b_desc_.p);
    a.cands = static_cast<CandRec*>(b_cands_.p);
    a.cap_specs = (u32)std::min<uint64_t>(0xFFFFFFF0u, std::min(b_hdrs_.cap / sizeof(SpecHdr), b_desc_.cap / sizeof(u64)));
    a.cap_cands = b_cands_.cap / sizeof(CandRec);
    a.phases = phases;
    CK(launch_plan_kernel(a, blocks(attempt == 0 ? tab.n_positions / 2 : want_specs), stream_));
    CK(cudaMemcpyAsync(h_stage_, res, back, cudaMemcpyDeviceToHost, stream_));
    CK(cudaStreamSynchronize(stream_));
    if (ctl->n_specs > 0xFFFFFFF0u || ctl->n_cands > 0xFFFFFFFFull || attempt > 4) return 1;
    want_specs = ctl->n_specs;
    want_cands = ctl->n_cands;
    if (ctl->n_specs > a.cap_specs || !b_hdrs_.p) phases = fixed_ ? DPP_SPECS : DPP_SPECS | DPP_RECORDS;
    else if (ctl->n_cands > a.cap_cands || !b_cands_.p || !(phases & DPP_RECORDS)) phases = DPP_RECORDS;
    else if (!fixed_ && (oversized_(b_hdrs_, want_specs * sizeof(SpecHdr)) || oversized_(b_desc_, want_specs * sizeof(u64)) ||
                         oversized_(b_cands_, want_cands * sizeof(CandRec)))) {   // of a far larger plan; the closure stays
      for (DevBuf* b : {&b_hdrs_, &b_desc_, &b_cands_}) drop_(*b);
      phases = DPP_SPECS | DPP_RECORDS;
    } else break;
    if (phases == DPP_RECORDS && (rc = reserve_(b_cands_, std::max<uint64_t>(want_cands, 1) * sizeof(CandRec), false))) return rc == -5 ? 1 : rc;
  }
  d_hdrs_ = a.hdrs;
  d_cands_ = a.cands;
  n_specs_ = ctl->n_specs;
  n_goals_ = ctl->n_goals;
  n_cand_bytes_ = ctl->n_cands * sizeof(CandRec);
  for (u32 g = 0; g < n_stages; g++)
    if (lo[g + 1] > lo[g]) {
      const u32 key = tab.stage_key[g];
      stages_.push_back(StageIds{lo[g], lo[g + 1], 0, team_of_stage(lo[g + 1] - lo[g], key >> 16, (key >> 8) & 0xFFu, key & 0xFFu)});
    }
  top_pack_ = 0;
  for (int k = 0; k < NMEM; k++) top_pack_ |= tab.top_code[k] << (8 * k);
  h2d_bytes_ = bytes;
  tab_.reset(new DevTables());
  tab_->t = a.t;
  stats_ = FillStats();
  return 0;
}

int DeviceFill::prepare_fill() {
  CK(cudaSetDevice(device_));
  int rc = working_buffers_(false, 1);
  if (rc == -6) {   // the ones of earlier plans may be in the way
    CK(cudaStreamSynchronize(stream_));
    for (DevBuf* b : {&b_items_, &b_temp_, &b_rows_, &b_lookup_, &b_bits_}) drop_(*b);
    rc = working_buffers_(false, 1);
  }
  if (rc) return rc;
  CK(cudaMemsetAsync(d_ctl_, 0, 512, stream_));
  cands_present_ = true;
  stats_ = FillStats();
  return 0;
}

int DeviceFill::sync() {
  CK(cudaStreamSynchronize(stream_));
  return 0;
}

int DeviceFill::cands_arrived() {
  CK(cudaSetDevice(device_));
  if (cands_present_) return 0;
  if (n_specs_) {
    check_records_kernel<<<(n_specs_ + kBlock - 1) / kBlock, kBlock, 0, stream_>>>(d_hdrs_, d_cands_, n_specs_,
                                                                                   n_cand_bytes_ / sizeof(CandRec), &d_ctl_->error);
    CK(cudaGetLastError());
  }
  if (read_ctl_() != 0) return -1;
  if (h_ctl_->error) {
    CK(cudaMemsetAsync(d_ctl_, 0, offsetof(FillCtl, failed_stage), stream_));   // the error, and what its stage had counted
    snprintf(err_, sizeof(err_), "the candidate records on the device do not describe this plan (a field is out of range)");
    return -2;
  }
  cands_present_ = true;
  return 0;
}

int DeviceFill::read_ctl_() {
  CK(cudaMemcpyAsync(h_ctl_, d_ctl_, sizeof(FillCtl), cudaMemcpyDeviceToHost, stream_));
  CK(cudaStreamSynchronize(stream_));
  return 0;
}

// After a stage asked for more room than a buffer had: enlarges what it named. Working buffers
// hold nothing worth keeping between stages; the rows placed so far move along.
int DeviceFill::grow_after_error_(uint32_t bits) {
  if (fixed_) return too_large_();
  stats_.growths++;
  CK(cudaStreamSynchronize(stream_));
  auto regrow = [&](DevBuf& b, uint64_t need, size_t elem) -> int {
    return need * elem <= b.cap ? 0 : reserve_(b, (need + need / 4) * elem);
  };
  int rc = 0;
  if (bits & MRL_ERR_WORKING) {
    if ((rc = regrow(b_temp_, h_ctl_->need_temp, 2 * sizeof(MrlRow))) == 0)
      rc = regrow(b_items_, h_ctl_->need_items, sizeof(WorkItem));
    temp_cap_ = b_temp_.cap / (2 * sizeof(MrlRow));
    item_cap_ = b_items_.cap / sizeof(WorkItem);
    d_temp_ = static_cast<MrlRow*>(b_temp_.p);
    d_items_ = static_cast<WorkItem*>(b_items_.p);
    if (rc) return rc;
  }
  if (bits & MRL_ERR_TABLE) {
    const uint64_t need = h_ctl_->need_rows;
    size_t free_b = 0, total_b = 0;
    CK(cudaMemGetInfo(&free_b, &total_b));
    uint64_t cap = std::max<uint64_t>(need + need / 8, row_cap_ * 2);
    if (cap * sizeof(MrlRow) + (1ull << 30) > free_b) cap = need + need / 16;
    MrlRow* nr = nullptr;
    if ((rc = alloc_((void**)&nr, cap * sizeof(MrlRow)))) {
      snprintf(err_, sizeof(err_), "out of device memory: the table needs %llu rows", (unsigned long long)need);
      return -6;
    }
    if (h_ctl_->final_top) CK(cudaMemcpyAsync(nr, d_rows_, h_ctl_->final_top * sizeof(MrlRow), cudaMemcpyDeviceToDevice, stream_));
    CK(cudaStreamSynchronize(stream_));
    drop_(b_rows_);
    b_rows_.p = d_rows_ = nr;
    b_rows_.cap = cap * sizeof(MrlRow);
    row_cap_ = cap;
  }
  return 0;
}

int DeviceFill::begin_fill() {
  CK(cudaSetDevice(device_));
  if (!cands_present_) {
    snprintf(err_, sizeof(err_), "the candidate records are not on the device yet (mrl_device_cands hands out the buffer; "
             "mrl_cands_arrived checks what was written)");
    return -3;
  }
  stats_ = FillStats();
  CK(cudaMemsetAsync(d_ctl_, 0, 512, stream_));
  CK(cudaEventRecord(ev0_, stream_));
  filling_ = true;
  return 0;
}

// One launch of the stage kernel for the stages [from, to), by a team that fits them (team_of_stage).
int DeviceFill::launch_stages_(uint32_t from, uint32_t to, int team, int blocks, bool solve, bool place) {
  StageArgs a;
  a.hdrs = d_hdrs_; a.cands = d_cands_; a.rmask = d_rmask_; a.mine = d_mine_; a.items = d_items_; a.rows = d_rows_; a.temp = d_temp_;
  a.minsat = d_minsat_; a.sspec = static_cast<StageSpec*>(d_sspec_);
  for (int k = 0; k < 3; k++) a.changed[k] = d_changed_[k];
  a.block_sums = d_block_sums_; a.ctl = d_ctl_; a.stages = static_cast<const uint2*>(b_stages_.p);
  a.stage_lo = from; a.stage_hi = to; a.top_pack = top_pack_; a.team = team;
  a.temp_cap = temp_cap_; a.item_cap = item_cap_; a.row_cap = row_cap_;
  a.solve = solve ? 1 : 0;
  a.place = place ? 1 : 0;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(kStageBlock);
  cfg.dynamicSmemBytes = kStageSmem;
  cfg.stream = stream_;
  cudaLaunchAttribute attr[1];
  if (team == TEAM_GRID) {
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
  } else {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = blocks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = team == TEAM_BLOCK ? 0 : 1;
  CK(cudaLaunchKernelEx(&cfg, stage_kernel, a));
  stats_.launches++;
  return 0;
}

int DeviceFill::blocks_of_(int team) const { return team == TEAM_BLOCK ? 1 : (team == TEAM_CLUSTER ? 8 : coop_blocks_); }

int DeviceFill::launch_solve_(uint32_t si, bool place_too) {
  const StageIds& st = stages_[si];
  if (st.hi == st.lo) return 0;
  // the stage reads its own Specs' candidate records (ids, and with them the records, are in
  // stage order): wait for that much of a background upload
  int rc = wait_cands_(st.cand_end * sizeof(CandRec));
  if (rc) return rc;
  return launch_stages_(si, si + 1, st.team, blocks_of_(st.team), true, place_too);
}

int DeviceFill::launch_place_(uint32_t si) {
  const StageIds& st = stages_[si];
  if (st.hi == st.lo) return 0;
  return launch_stages_(si, si + 1, st.team, blocks_of_(st.team), false, true);
}

int DeviceFill::solve_stage(uint32_t si) {
  if (si >= stages_.size()) { snprintf(err_, sizeof(err_), "stage index out of range"); return -3; }
  if (!filling_) { snprintf(err_, sizeof(err_), "no fill in progress"); return -3; }
  return launch_solve_(si, false);
}

static const char* kErrorBits = "(1: candidate record out of range, 2: working buffers too small, 4: row table too small, "
                                "8: no consistent limits grid)";

// Where the stage's real-breakpoint masks lie (what the ranks exchange before any of them places
// the stage). The masks must be final before they travel, so this is where a rank learns that its
// solve ran out of working room: it enlarges its own buffers and solves the stage again; the other
// ranks wait in the exchange.
int DeviceFill::stage_masks(uint32_t si, void** ptr, uint64_t* bytes) {
  if (si >= stages_.size()) { snprintf(err_, sizeof(err_), "stage index out of range"); return -3; }
  const StageIds& st = stages_[si];
  if (filling_ && st.hi != st.lo) {
    int rc;
    if (read_ctl_() != 0) return -1;
    if (h_ctl_->error & MRL_ERR_WORKING) {
      const uint32_t bits = h_ctl_->error;
      if (bits & ~(uint32_t)(MRL_ERR_WORKING | MRL_ERR_TABLE)) {
        snprintf(err_, sizeof(err_), "a fill kernel reported error bits 0x%x in stage %u %s", bits, h_ctl_->failed_stage, kErrorBits);
        return -2;
      }
      if ((rc = grow_after_error_(MRL_ERR_WORKING))) return rc;
      CK(cudaMemsetAsync(d_ctl_, 0, offsetof(FillCtl, failed_stage), stream_));   // the error, and what its stage had counted
      if ((rc = launch_solve_(si, false))) return rc;
      if (read_ctl_() != 0) return -1;
      if (h_ctl_->error) {
        snprintf(err_, sizeof(err_), "stage %u failed again after its working buffers were enlarged (0x%x)", si, h_ctl_->error);
        return -2;
      }
    }
  }
  if (ptr) *ptr = d_rmask_ + st.lo;
  if (bytes) *bytes = (uint64_t)(st.hi - st.lo) * sizeof(uint4);
  return 0;
}

// Appends the stage's compacted grids to the table and reports where they went (the slice other
// ranks need), which costs the one synchronisation of the stage. A stage that ran out of room is
// run again here, whole, after its buffers have grown: its masks cannot have been exchanged yet.
int DeviceFill::place_stage(uint32_t si, void** rows_ptr, uint64_t* bytes) {
  if (si >= stages_.size()) { snprintf(err_, sizeof(err_), "stage index out of range"); return -3; }
  if (!filling_) { snprintf(err_, sizeof(err_), "no fill in progress"); return -3; }
  if (rows_ptr) *rows_ptr = d_rows_;
  if (bytes) *bytes = 0;
  const StageIds& st = stages_[si];
  if (st.hi == st.lo) return 0;
  int rc;
  if ((rc = launch_place_(si))) return rc;
  if (read_ctl_() != 0) return -1;
  if (h_ctl_->error) {
    const uint32_t bits = h_ctl_->error;
    if (bits & MRL_ERR_WORKING) {
      snprintf(err_, sizeof(err_), "stage %u needs larger working buffers than a sharded fill starts with "
               "(%llu working rows); fill once unsharded, or with fewer Specs per stage", si,
               (unsigned long long)h_ctl_->need_temp);
      return -6;
    }
    if (bits & ~(uint32_t)MRL_ERR_TABLE) {
      snprintf(err_, sizeof(err_), "a fill kernel reported error bits 0x%x in stage %u %s", bits, h_ctl_->failed_stage, kErrorBits);
      return -2;
    }
    if ((rc = grow_after_error_(bits))) return rc;
    CK(cudaMemsetAsync(d_ctl_, 0, offsetof(FillCtl, failed_stage), stream_));   // the error, and what its stage had counted
    if ((rc = launch_place_(si))) return rc;
    if (read_ctl_() != 0) return -1;
    if (h_ctl_->error) { snprintf(err_, sizeof(err_), "stage %u failed again after its buffers were enlarged (0x%x)", si, h_ctl_->error); return -2; }
  }
  if (rows_ptr) *rows_ptr = d_rows_ + h_ctl_->stage_first_row;
  if (bytes) *bytes = h_ctl_->stage_rows * sizeof(MrlRow);
  return 0;
}

void DeviceFill::take_stats_() {
  const FillCtl& c = *h_ctl_;
  stats_.n_rows = c.final_top;
  stats_.cells_solved = c.st_cells;
  stats_.cands_evaluated = c.st_cands;
  stats_.lookups = c.st_lookups;
  stats_.alg_bytes = c.st_final_bytes;
  stats_.passes = c.st_passes;
  stats_.grid_syncs = c.st_syncs;
  stats_.sweeps = c.st_sweeps;
  stats_.early_cells = c.st_early_cells;
  stats_.late_cands = c.st_late_cands;
  stats_.late_items = c.st_late_items;
  for (int k = 0; k < 8; k++) stats_.phase_ms[k] = (float)(c.st_phase_ns[k] * 1e-6);
  stats_.early_ms = stats_.phase_ms[MRL_PH_EARLY];
  stats_.combine_ms = stats_.early_ms + stats_.phase_ms[MRL_PH_INIT] + stats_.phase_ms[MRL_PH_SWEEP_FIRST] + stats_.phase_ms[MRL_PH_SWEEP_MORE];
}

int DeviceFill::end_fill() {
  CK(cudaEventRecord(ev1_, stream_));
  if (read_ctl_() != 0) return -1;
  filling_ = false;
  CK(cudaEventElapsedTime(&stats_.fill_ms, ev0_, ev1_));
  take_stats_();
  if (h_ctl_->error) {
    snprintf(err_, sizeof(err_), "a fill kernel reported error bits 0x%x in stage %u %s", h_ctl_->error, h_ctl_->failed_stage, kErrorBits);
    return -2;
  }
  return 0;
}

// Every stage is enqueued without waiting for the one before: sizes, pass counts and launch
// geometry are all decided on the device. A stage that runs out of room raises an error word
// that turns the stages behind it into no-ops; the host then enlarges the buffers it named and
// resumes from that stage.
int DeviceFill::run() {
  int rc;
  if ((rc = begin_fill())) return rc;
  uint32_t from = 0;
  for (int attempt = 0;; attempt++) {
    // Consecutive stages with the same team run as one launch: a launch of its own costs a stage 20 us
    // (gap, cold instruction and data caches) where a small one takes 15 (2x8x4 Matmul in both dtypes,
    // 40 k Specs in 141 stages: 14.8 -> 12.3 ms together with the teams). In plans of more than
    // kMergeSpecs that is 2 % or less (precompute 4, 642 k Specs: 28.3 -> 27.7 ms), and a launch per stage
    // is what their statistics and profiles are read by. While candidate records are still on their way
    // up, every stage waits for its own.
    for (uint32_t s = from, e; s < stages_.size(); s = e) {
      e = s + 1;
      if (n_specs_ <= kMergeSpecs && up_threads_.empty())
        while (e < stages_.size() && stages_[e].team == stages_[s].team) e++;
      if (e == s + 1) rc = launch_solve_(s, true);
      else rc = launch_stages_(s, e, stages_[s].team, blocks_of_(stages_[s].team), true, true);
      if (rc) return rc;
    }
    CK(cudaEventRecord(ev1_, stream_));
    if (read_ctl_() != 0) return -1;
    const uint32_t bits = h_ctl_->error;
    if (!bits) break;
    if ((bits & ~(uint32_t)(MRL_ERR_WORKING | MRL_ERR_TABLE)) || attempt >= 64) {
      filling_ = false;
      take_stats_();
      snprintf(err_, sizeof(err_), "a fill kernel reported error bits 0x%x in stage %u %s", bits, h_ctl_->failed_stage, kErrorBits);
      return -2;
    }
    from = h_ctl_->failed_stage;
    if ((rc = grow_after_error_(bits))) { filling_ = false; return rc; }
    CK(cudaMemsetAsync(d_ctl_, 0, offsetof(FillCtl, failed_stage), stream_));   // the error, and what its stage had counted
  }
  filling_ = false;
  CK(cudaEventElapsedTime(&stats_.fill_ms, ev0_, ev1_));
  take_stats_();
  return 0;
}

// Point lookups: the queries go up from pinned staging and the rows come back into it, in batches.
template <class Fill, class Launch>
int DeviceFill::lookup_batches_(size_t n, size_t query_bytes, MrlRow* out, Fill fill, Launch launch) {
  const size_t per = std::max(query_bytes, sizeof(MrlRow));
  size_t batch = std::min<size_t>(n, size_t(1) << 20);
  if (fixed_) batch = std::min(n, b_lookup_.cap / 2 / per);
  else {
    int rc = reserve_(b_lookup_, 2 * align256(batch * per));
    if (rc) return rc;
  }
  if (batch == 0) { snprintf(err_, sizeof(err_), "lookup staging too small"); return -5; }
  int rc = reserve_host_(batch * per);
  if (rc) return rc;
  unsigned char* const d_q = static_cast<unsigned char*>(b_lookup_.p);
  MrlRow* const d_out = reinterpret_cast<MrlRow*>(d_q + b_lookup_.cap / 2 / 256 * 256);
  for (size_t done = 0; done < n; done += batch) {
    const size_t m = std::min(batch, n - done);
    fill(h_stage_, done, m);
    CK(cudaMemcpyAsync(d_q, h_stage_, m * query_bytes, cudaMemcpyHostToDevice, stream_));
    launch(d_q, m, d_out);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(h_stage_, d_out, m * sizeof(MrlRow), cudaMemcpyDeviceToHost, stream_));
    CK(cudaStreamSynchronize(stream_));
    memcpy(out + done, h_stage_, m * sizeof(MrlRow));
  }
  return 0;
}

int DeviceFill::lookup(const uint32_t* spec_ids, const uint32_t* cpacks, size_t n, MrlRow* out) {
  std::lock_guard<std::mutex> guard(lookup_mu_);   // callers on several threads share the staging buffers and the stream
  CK(cudaSetDevice(device_));
  if (n == 0) return 0;
  for (size_t i = 0; i < n; i++)
    if (spec_ids[i] >= n_specs_) { snprintf(err_, sizeof(err_), "Spec id out of range"); return -3; }
  return lookup_batches_(n, sizeof(uint2), out,
                         [&](void* to, size_t at, size_t m) {
                           uint2* q = static_cast<uint2*>(to);
                           for (size_t i = 0; i < m; i++) q[i] = make_uint2(spec_ids[at + i], cpacks[at + i]);
                         },
                         [&](const void* q, size_t m, MrlRow* d_out) {
                           lookup_rows_kernel<<<(unsigned)((m + kBlock - 1) / kBlock), kBlock, 0, stream_>>>(
                               d_hdrs_, d_rows_, static_cast<const uint2*>(q), m, d_out);
                         });
}

int DeviceFill::lookup_packed(const uint64_t* specs, const uint32_t* cpacks, size_t n, MrlRow* out) {
  std::lock_guard<std::mutex> guard(lookup_mu_);
  CK(cudaSetDevice(device_));
  if (n == 0) return 0;
  if (!tab_) { snprintf(err_, sizeof(err_), "no plan made on the device"); return -3; }
  return lookup_batches_(n, sizeof(PackedQuery), out,
                         [&](void* to, size_t at, size_t m) {
                           PackedQuery* q = static_cast<PackedQuery*>(to);
                           for (size_t i = 0; i < m; i++) q[i] = PackedQuery{specs[at + i], cpacks[at + i], 0u};
                         },
                         [&](const void* q, size_t m, MrlRow* d_out) {
                           lookup_packed_kernel<<<(unsigned)((m + kBlock - 1) / kBlock), kBlock, 0, stream_>>>(
                               tab_->t, d_hdrs_, d_rows_, static_cast<const PackedQuery*>(q), m, d_out);
                         });
}

int DeviceFill::walk(uint64_t root, bool packed, uint32_t cpack, std::vector<WalkNode>& out) {
  std::lock_guard<std::mutex> guard(lookup_mu_);
  CK(cudaSetDevice(device_));
  if (packed && !tab_) { snprintf(err_, sizeof(err_), "no plan made on the device"); return -3; }
  if (wait_upload()) return -1;   // a table that was loaded may be here before the records are
  const size_t head = align256(sizeof(uint32_t)), bytes = head + kWalkMost * sizeof(WalkNode), first = head + 96 * sizeof(WalkNode);
  int rc;
  if ((rc = reserve_(b_lookup_, bytes, false)) || (rc = reserve_host_(bytes))) return rc;
  unsigned char* const d = static_cast<unsigned char*>(b_lookup_.p);
  DpTables t;
  memset(&t, 0, sizeof(t));
  if (tab_) t = tab_->t;
  walk_kernel<<<1, kBlock, 0, stream_>>>(t, tab_ ? static_cast<const unsigned long long*>(b_desc_.p) : nullptr, d_hdrs_, d_cands_, d_rows_, n_specs_,
                                         root, packed ? 1u : 0u, cpack, reinterpret_cast<WalkNode*>(d + head), reinterpret_cast<uint32_t*>(d));
  CK(cudaGetLastError());
  unsigned char* const h = static_cast<unsigned char*>(h_stage_);
  CK(cudaMemcpyAsync(h, d, first, cudaMemcpyDeviceToHost, stream_));   // most trees are smaller than this
  CK(cudaStreamSynchronize(stream_));
  const uint32_t n = *reinterpret_cast<const uint32_t*>(h);
  if (n > kWalkMost) return 1;
  if (head + n * sizeof(WalkNode) > first) {
    CK(cudaMemcpyAsync(h + first, d + first, head + n * sizeof(WalkNode) - first, cudaMemcpyDeviceToHost, stream_));
    CK(cudaStreamSynchronize(stream_));
  }
  const WalkNode* const nodes = reinterpret_cast<const WalkNode*>(h + head);
  out.assign(nodes, nodes + n);
  return 0;
}

// Device memory into pageable memory of the caller's, which is often fresh: the driver's own staging
// runs on one thread, and half of its time goes into page faults. Large parts are brought over in
// pieces by a few threads, each through two pinned buffers of its own. Pinning them is most of a database's
// first export: 57 MB of rows take 14 ms the first time and 5.8 then with pieces of 1 MB, 20 and 5.7 with 2 MB,
// 13 and 6.7 with 512 KB.
int DeviceFill::read_bulk_(void* out, const void* src, size_t bytes) {
  const size_t piece = size_t(1) << 20;
  const int n_threads = 4;
  if (bytes < 8 * piece || fixed_ || reserve_host_(n_threads * 2 * piece) != 0) {
    cudaGetLastError();   // no pinned memory to be had is no reason to refuse
    if (bytes) CK(cudaMemcpyAsync(out, src, bytes, cudaMemcpyDeviceToHost, stream_));
    CK(cudaStreamSynchronize(stream_));
    return 0;
  }
  CK(cudaStreamSynchronize(stream_));
  std::atomic<size_t> next{0};
  std::atomic<int> error{0};
  const size_t pieces = (bytes + piece - 1) / piece;
  auto work = [&](int t) {
    unsigned char* const pin = static_cast<unsigned char*>(h_stage_) + (size_t)t * 2 * piece;
    cudaStream_t st = nullptr;
    cudaEvent_t ev[2] = {nullptr, nullptr};
    cudaError_t e = cudaSetDevice(device_);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    for (int b = 0; b < 2 && e == cudaSuccess; b++) e = cudaEventCreateWithFlags(&ev[b], cudaEventDisableTiming);
    size_t at[2] = {pieces, pieces};   // piece under way in each buffer
    for (int b = 0; e == cudaSuccess; b ^= 1) {
      if (at[b] < pieces) {
        e = cudaEventSynchronize(ev[b]);
        if (e != cudaSuccess) break;
        memcpy(static_cast<unsigned char*>(out) + at[b] * piece, pin + b * piece, std::min(piece, bytes - at[b] * piece));
        at[b] = pieces;
      }
      const size_t k = next.fetch_add(1);
      if (k < pieces) {
        at[b] = k;
        e = cudaMemcpyAsync(pin + b * piece, static_cast<const unsigned char*>(src) + k * piece, std::min(piece, bytes - k * piece),
                            cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaEventRecord(ev[b], st);
      } else if (at[b ^ 1] >= pieces) {
        break;
      }
    }
    if (st) { cudaStreamSynchronize(st); cudaStreamDestroy(st); }
    for (cudaEvent_t v : ev) if (v) cudaEventDestroy(v);
    if (e != cudaSuccess) error.store((int)e);
  };
  on_threads(n_threads, work);
  CK((cudaError_t)error.load());
  return 0;
}

int DeviceFill::export_table(uint32_t* masks, uint64_t* first_row, MrlRow* rows) {
  std::lock_guard<std::mutex> guard(lookup_mu_);   // the pinned staging is the lookups'
  CK(cudaSetDevice(device_));
  if (n_specs_) {
    const size_t o_first = align256((size_t)n_specs_ * sizeof(uint4)), need = o_first + (size_t)n_specs_ * sizeof(uint64_t);
    // the working rows are idle between fills
    if (b_temp_.cap < need) {
      int rc = reserve_(b_lookup_, need, false);
      if (rc) return rc;
    }
    unsigned char* const d = static_cast<unsigned char*>(b_temp_.cap >= need ? b_temp_.p : b_lookup_.p);
    export_headers_kernel<<<(n_specs_ + kBlock - 1) / kBlock, kBlock, 0, stream_>>>(d_hdrs_, n_specs_, reinterpret_cast<uint4*>(d),
                                                                                    reinterpret_cast<unsigned long long*>(d + o_first));
    CK(cudaGetLastError());
    int rc;
    if ((rc = read_bulk_(masks, d, (size_t)n_specs_ * sizeof(uint4))) || (rc = read_bulk_(first_row, d + o_first, (size_t)n_specs_ * sizeof(uint64_t))))
      return rc;
  }
  return read_bulk_(rows, d_rows_, stats_.n_rows * sizeof(MrlRow));
}

int DeviceFill::read_specs(uint64_t* out) {
  CK(cudaSetDevice(device_));
  if (!tab_) { snprintf(err_, sizeof(err_), "no plan made on the device"); return -3; }
  CK(cudaMemcpyAsync(out, b_desc_.p, (size_t)n_specs_ * sizeof(uint64_t), cudaMemcpyDeviceToHost, stream_));
  CK(cudaStreamSynchronize(stream_));
  return 0;
}

int DeviceFill::read_hdrs(SpecHdr* out) {
  CK(cudaSetDevice(device_));
  if (n_specs_) CK(cudaMemcpyAsync(out, d_hdrs_, (size_t)n_specs_ * sizeof(SpecHdr), cudaMemcpyDeviceToHost, stream_));
  CK(cudaStreamSynchronize(stream_));
  return 0;
}

// Checks the finished table against its defining recurrence at n_samples pseudo-random points of
// (Spec x limits lattice), or at every point when n_samples == 0.
int DeviceFill::verify(uint64_t n_samples, uint64_t seed, uint64_t* checked, uint64_t* mismatches,
                       uint64_t* first_bad) {
  CK(cudaSetDevice(device_));
  if (wait_upload()) return -1;
  const uint32_t top = top_pack_;
  unsigned long long per_spec = 1;
  for (int k = 0; k < 4; k++) per_spec *= ((top >> (8 * k)) & 0xFFu) + 1u;
  const unsigned long long total = per_spec * n_specs_;
  const bool exhaustive = n_samples == 0;
  const unsigned long long count = exhaustive ? total : n_samples;
  unsigned long long* d_out = d_ctl_->scratch;
  const unsigned long long init[2] = {0ull, ~0ull};
  CK(cudaMemcpyAsync(d_out, init, sizeof(init), cudaMemcpyHostToDevice, stream_));
  CK(cudaStreamSynchronize(stream_));
  const unsigned long long batch = 1ull << 28;
  for (unsigned long long first = 0; first < count && total; first += batch) {
    const unsigned long long n = std::min(batch, count - first);
    verify_points_kernel<<<(unsigned)((n + kBlock - 1) / kBlock), kBlock, 0, stream_>>>(d_hdrs_, d_cands_, d_rows_, n_specs_, top, first, n,
                                                                                       total, seed, exhaustive ? 1 : 0, d_out);
    CK(cudaGetLastError());
  }
  unsigned long long res[2] = {0, 0};
  CK(cudaMemcpyAsync(res, d_out, sizeof(res), cudaMemcpyDeviceToHost, stream_));
  CK(cudaStreamSynchronize(stream_));
  if (checked) *checked = total ? count : 0;
  if (mismatches) *mismatches = res[0];
  if (first_bad) *first_bad = res[1];
  return 0;
}

int DeviceFill::checksum(uint64_t* out) {
  CK(cudaSetDevice(device_));
  unsigned long long* d_out = d_ctl_->scratch + 2;
  CK(cudaMemsetAsync(d_out, 0, sizeof(unsigned long long), stream_));
  if (n_specs_) {
    checksum_kernel<<<(n_specs_ + kBlock - 1) / kBlock, kBlock, 0, stream_>>>(d_hdrs_, d_rows_, n_specs_, d_out);
    CK(cudaGetLastError());
  }
  unsigned long long v = 0;
  CK(cudaMemcpyAsync(&v, d_out, sizeof(v), cudaMemcpyDeviceToHost, stream_));
  CK(cudaStreamSynchronize(stream_));
  *out = v;
  return 0;
}

int DeviceFill::read_table(SpecHdr* hdrs_out, MrlRow* rows_out) {
  CK(cudaSetDevice(device_));
  if (n_specs_) CK(cudaMemcpyAsync(hdrs_out, d_hdrs_, (size_t)n_specs_ * sizeof(SpecHdr), cudaMemcpyDeviceToHost, stream_));
  if (stats_.n_rows) CK(cudaMemcpyAsync(rows_out, d_rows_, stats_.n_rows * sizeof(MrlRow), cudaMemcpyDeviceToHost, stream_));
  CK(cudaStreamSynchronize(stream_));
  return 0;
}

int DeviceFill::load_table(const SpecHdr* hdrs, const MrlRow* rows, uint64_t n_rows) {
  CK(cudaSetDevice(device_));
  if (n_rows > row_cap_) {
    if (fixed_) return too_large_();
    int rc = reserve_(b_rows_, n_rows * sizeof(MrlRow));
    d_rows_ = static_cast<MrlRow*>(b_rows_.p);
    row_cap_ = b_rows_.cap / sizeof(MrlRow);
    if (rc) return rc;
  }
  if (n_specs_) CK(cudaMemcpyAsync(d_hdrs_, hdrs, (size_t)n_specs_ * sizeof(SpecHdr), cudaMemcpyHostToDevice, stream_));
  if (n_rows) CK(cudaMemcpyAsync(d_rows_, rows, n_rows * sizeof(MrlRow), cudaMemcpyHostToDevice, stream_));
  CK(cudaStreamSynchronize(stream_));
  stats_ = FillStats();
  stats_.n_rows = n_rows;
  return 0;
}

int DeviceFill::read_hdr(uint32_t spec, SpecHdr* out) {
  CK(cudaSetDevice(device_));
  if (spec >= n_specs_) { snprintf(err_, sizeof(err_), "Spec id out of range"); return -3; }
  CK(cudaMemcpyAsync(out, d_hdrs_ + spec, sizeof(SpecHdr), cudaMemcpyDeviceToHost, stream_));
  CK(cudaStreamSynchronize(stream_));
  return 0;
}

int DeviceFill::read_rows(uint64_t first, uint64_t n, MrlRow* out) {
  CK(cudaSetDevice(device_));
  if (first + n > stats_.n_rows) { snprintf(err_, sizeof(err_), "row range out of the table"); return -3; }
  if (n == 0) return 0;
  CK(cudaMemcpyAsync(out, d_rows_ + first, n * sizeof(MrlRow), cudaMemcpyDeviceToHost, stream_));
  CK(cudaStreamSynchronize(stream_));
  return 0;
}

// ---------------------------------------------------------------------------------------
// Fill without device allocation.
//
// Some callers of this library must not allocate device memory while they run: a host that
// reserved all of HBM for its replicated tables at start-up has nothing left to hand out, and
// a worker pool that calls top_down_many from many threads would be serialised by the
// device-wide synchronisation every cudaMalloc / cudaFree implies. For them the whole device
// working set of one small fill - plan arrays, working buffers, row table, lookup staging - is
// carved out of the fixed array below instead of being allocated per call. Every GPU that
// loads this library holds the array until the process exits.
//
// In host code `g_static_scratch` is only a stand-in for the device array, not a device
// address; the address a kernel may use comes from cudaGetSymbolAddress, asked once per
// device with that device current (static_scratch_address).
namespace {
__device__ __align__(256) unsigned char g_static_scratch[MRL_STATIC_SCRATCH_BYTES];

constexpr int kMaxDevices = 64;
void* g_scratch_addr[kMaxDevices] = {nullptr};
std::mutex g_scratch_mu;

// Device address of the static array on `device`, resolved on first use. The caller's current
// device is left as it was.
cudaError_t static_scratch_address(int device, void** out) {
  if (device < 0 || device >= kMaxDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> g(g_scratch_mu);
  if (!g_scratch_addr[device]) {
    int before = -1;
    cudaError_t e = cudaGetDevice(&before);
    if (e != cudaSuccess) return e;
    e = cudaSetDevice(device);
    if (e != cudaSuccess) return e;
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_static_scratch);
    if (before != device) cudaSetDevice(before);
    if (e != cudaSuccess) return e;
    g_scratch_addr[device] = p;
  }
  *out = g_scratch_addr[device];
  return cudaSuccess;
}
}  // namespace

// Runs `plan` entirely inside the static array and copies the rows of the given (Spec id,
// packed limit codes) queries to `out` (host). No cudaMalloc / cudaFree. Returns -5 with a
// message when the fill does not fit.
int fill_static(int device, cudaStream_t stream, const Plan& plan, const uint32_t* spec_ids, const uint32_t* cpacks,
                size_t n, MrlRow* out, char* err, size_t err_len) {
  void* base = nullptr;
  cudaError_t e = static_scratch_address(device, &base);
  if (e == cudaSuccess) e = cudaSetDevice(device);
  if (e != cudaSuccess) {
    snprintf(err, err_len, "static scratch unavailable: %s", cudaGetErrorString(e));
    return -1;
  }
  DeviceFill f;
  f.attach_buffer(base, (size_t)MRL_STATIC_SCRATCH_BYTES, stream, device);
  int rc = f.init_events();
  if (rc == 0) rc = f.upload(plan);
  if (rc == 0) rc = f.run();
  if (rc == 0) rc = f.lookup(spec_ids, cpacks, n, out);
  if (rc != 0) snprintf(err, err_len, "%s", f.error());
  return rc;
}

int fill_static(int device, cudaStream_t stream, const OpTables& tab, const uint64_t* specs, const uint32_t* cpacks,
                size_t n, MrlRow* out, char* err, size_t err_len) {
  void* base = nullptr;
  cudaError_t e = static_scratch_address(device, &base);
  if (e == cudaSuccess) e = cudaSetDevice(device);
  if (e != cudaSuccess) {
    snprintf(err, err_len, "static scratch unavailable: %s", cudaGetErrorString(e));
    return -1;
  }
  DeviceFill f;
  f.attach_buffer(base, (size_t)MRL_STATIC_SCRATCH_BYTES, stream, device);
  int rc = f.init_events();
  if (rc == 0) rc = f.plan(tab);
  if (rc == 0) rc = f.prepare_fill();
  if (rc == 0) rc = f.run();
  if (rc == -5) rc = 1;   // the plan's tables take a little room of their own: without them it may fit
  if (rc == 0) rc = f.lookup_packed(specs, cpacks, n, out);
  if (rc < 0) snprintf(err, err_len, "%s", f.error());
  return rc;
}

}  // namespace mrl
