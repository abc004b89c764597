// Plain-data records shared by the host planner and the CUDA fill kernels.
//
// Limits lattice: one integer "code" per memory, in the reference's own database
// coordinates (MemoryLimitsBimap, morello/src/memorylimits.rs:696-734): registers (RF, VRF)
// use the raw count, caches (L1, GL) use the bit length of the line count (0 -> 0,
// 2^(c-1) lines -> c).
#pragma once
#include <stdint.h>

// One table row = the optimum of one (logical Spec, limits cell): the reference's
// (ActionNum, Cost{main, peaks, depth}) (morello/src/db/mod.rs:54,171; morello/src/cost.rs:13-17).
// Compared as the 96-bit big-endian number (main, peaks, tail) it orders exactly like
// (Cost, ActionNum) (morello/src/cost.rs:87-104, morello/src/search/reducer.rs:41-48);
// an unsatisfiable cell is all ones, which sorts after everything.
struct MrlRow {
  uint32_t main;   // saturating u32 main cost
  uint32_t peaks;  // RF<<24 | VRF<<16 | L1 code<<8 | GL code   (peak memory, as lattice codes)
  uint32_t tail;   // depth<<16 | action number; 0xFFFFFFFF = no implementation
  uint32_t aux;    // 0 (1 in a lookup's answer for a Spec that does not exist).
                   // 12 bytes of payload in a 16-byte slot: one aligned vector load per gather.
};
#define MRL_UNSAT 0xFFFFFFFFu

// Per logical Spec: breakpoint masks of its limits grid (bit c set = code c starts a new
// cell; bit 0 always set), the first row of its dense cell block and its candidates.
// Cell (i0,i1,i2,i3) has row ((i3*n2 + i2)*n1 + i1)*n0 + i0 with n_k = popcount(mask[k]).
// While a stage is being solved its Specs point at a working grid in the working-row buffer;
// once the stage is consistent they point at the compacted final grid.
struct SpecHdr {
  uint32_t mask[4];
  uint64_t row_base;
  uint32_t cand_off;
  uint32_t ncand;
};

enum { MRL_CK_LEAF = 0, MRL_CK_LOOP = 1, MRL_CK_MOVE = 2, MRL_CK_BLOCK = 3 };

// One applicable action of a Spec, reduced to what the limits-dependent combine needs
// (morello/src/scheduling/mod.rs:286-368).
struct CandRec {
  uint16_t action;   // ActionNum in the reference's enumeration order
  uint8_t kind;      // MRL_CK_*
  uint8_t nchild;    // 0..3
  uint32_t imm;      // LEAF: kernel main cost; LOOP: iterations; MOVE: base move cost
  uint8_t level;     // memory the action allocates in (MOVE, LEAF)
  uint8_t thr_code;  // smallest limit code in `level` at which the action applies
  uint8_t peak_code; // LEAF: the kernel's own peak in `level`, as a code
  uint8_t late;      // 1: a child lies in the Spec's own stage (a relayout Move); such records come last
  uint32_t units;    // MOVE: units consumed in `level` (registers or cache lines)
  uint32_t child[3]; // Spec ids, in request order
  uint32_t pad1;
};

// A piece of one Spec's grid for a solve phase: consecutive cells from
// first_cell on, at most MRL_ITEM_CELLS of them (the stage kernel picks the size, 32 << bits 1 to 3 of
// first_cell; bit 0: the grid is new in this pass). Warps take items as they finish others.
#define MRL_ITEM_CELLS 1024u
struct WorkItem {
  uint32_t spec;
  uint32_t first_cell;
};

// What the stage kernel keeps per Spec of the stage being solved.
#ifdef __CUDACC__
struct __align__(16) StageSpec {
  uint4 emask;         // grid of the unordered phase
  uint4 old_mask;      // working grid before it last grew, and its rows
  unsigned long long erow;      // first row of the grid of the unordered phase
  unsigned long long old_row;
  uint32_t corner;     // where its grids are clipped
  uint32_t n_late;     // records with a same-stage child
  uint32_t dirty;      // its working grid grew or changed in this pass
  uint32_t pad;
};
#endif
#define MRL_STAGE_SPEC_BYTES 64u

// Error bits a fill kernel can raise (sticky until the host clears them).
enum {
  MRL_ERR_CHILD = 1,      // a candidate record names a Spec id outside the plan
  MRL_ERR_WORKING = 2,    // a working buffer (rows, chunks, work items) is too small
  MRL_ERR_TABLE = 4,      // the row table is too small
  MRL_ERR_PASSES = 8,     // a stage did not reach a consistent limits grid
};

// Parts of a stage kernel whose device time is accounted separately.
enum {
  MRL_PH_SETUP = 0,       // corners, grids of the unordered phase, their placement
  MRL_PH_EARLY = 1,       // the unordered phase
  MRL_PH_EARLY_MASKS = 2, // real breakpoints of its result
  MRL_PH_PASS_SETUP = 3,  // per pass: working grids, marks, placement
  MRL_PH_INIT = 4,        // per pass: cells start from the unordered phase's result
  MRL_PH_SWEEP_FIRST = 5, // per pass: the first relaxation sweep
  MRL_PH_SWEEP_MORE = 6,  // per pass: the sweeps after it
  MRL_PH_PASS_MASKS = 7,  // per pass: real breakpoints of the working grids
};

// Control block of a fill, in device memory. The stage kernels read their sizes and cursors
// here and leave the host nothing to decide between launches; the host reads it once per fill
// (once per stage when the fill is sharded).
struct StageCtl {                    // of one stage; zero at its start
  unsigned long long rows_early;     // rows handed out to the grids of the unordered phase
  unsigned long long rows_late;      // working rows handed out
  uint32_t n_items_early;            // work items listed for the grids of the unordered phase
  uint32_t n_items;                  // ... for the working grids. A word of its own: a stage whose unordered phase left
                                     // no items adds to it while slower threads still read how many that phase left
  uint32_t any_late;                 // stage + 1 when some Spec of it has a record with a same-stage child
  uint32_t any_changed;              // last relaxation sweep that changed a cell; only grows within a stage
  uint32_t grew;                     // pass + 1 when a grid has to grow after it
  uint32_t next_item[8];             // item hand-out of a phase; the phases take turns
};
// Whether a relaxation sweep changed a cell, from StageCtl::any_changed as read behind the sweep's barrier.
// Nothing separates that read from the next sweep of the threads that have made it already, so the word may
// hold the next sweep's number by then - which is only ever stored where this one changed something.
#ifdef __CUDACC__
__host__ __device__
#endif
inline bool sweep_changed_a_cell(uint32_t any_changed, uint32_t sweep) { return any_changed >= sweep; }

struct FillCtl {
  StageCtl stage;
  // -- sticky over a fill
  uint32_t error;                    // MRL_ERR_* bits
  uint32_t failed_stage;             // first stage that raised one
  unsigned long long need_temp, need_items, need_rows;   // what it would have taken
  unsigned long long final_top;      // rows of the finished table
  unsigned long long stage_first_row, stage_rows;   // the last placed stage's slice of the table
  // -- statistics of a fill
  unsigned long long st_cells;       // working cells solved, all passes
  unsigned long long st_cands;       // candidate records evaluated
  unsigned long long st_lookups;     // child rows gathered
  unsigned long long st_passes;
  unsigned long long st_final_bytes; // algorithmic bytes of the finished rows (see fill.hpp)
  unsigned long long st_syncs;       // barriers of a stage's team executed (a grid, a cluster or a block)
  unsigned long long st_sweeps;      // relaxation sweeps, all passes
  unsigned long long st_early_cells; // of st_cells: cells of the grids of the unordered phase
  unsigned long long st_late_cands;  // of st_cands: evaluated by the sweeps
  unsigned long long st_late_items;  // work items the sweeps evaluated
  unsigned long long st_phase_ns[8]; // device time by part of the stage kernel (see MRL_PH_*)
  // -- scratch of verify and checksum
  unsigned long long scratch[4];
};

#ifdef __cplusplus
static_assert(sizeof(MrlRow) == 16, "row slot is 16 bytes");
static_assert(sizeof(SpecHdr) == 32, "spec header is 32 bytes");
static_assert(sizeof(CandRec) == 32, "candidate record is 32 bytes");
static_assert(sizeof(FillCtl) % 8 == 0 && sizeof(FillCtl) <= 512, "control block");
#endif
