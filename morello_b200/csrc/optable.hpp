// The factored form of a planning job, from which the device works out the whole plan.
//
// What a candidate action does to a Spec it does operand by operand: a Move replaces one operand's
// aux, a tile-out or split replaces every operand by its tile. So instead of tabulating Specs, the
// host interns OPERANDS (shape and aux; 15 of them for a 2x2x2 Matmul, 4 918 for a size-8
// precompute against 7.3 M Specs) and tabulates, per operand, its Moves and its tiles. A Spec is a
// family (dtype, kind, shape) and one operand index per position, and everything about it - its
// place in the id order, its candidates, their children - is arithmetic on these tables
// (devplan.cu).
//
// Id order without a sort: ids are stage-major, then in key order (plan.cpp, "final ids"). A key
// is the family's bytes followed by each operand's bytes, and no operand encoding is a prefix of
// another one, so key order is (family bytes, operand 0, operand 1, operand 2) with operands of a
// shape numbered in byte order. Every (family, memory-level rank) gets a dense slice of positions,
// slices laid out in id order; a bitmap over the positions says which Specs exist, and a Spec's id
// is the number of bits set before its own.
#pragma once
#include "plan.hpp"
#include "model/actions.hpp"
#include <vector>

namespace mrl {

struct DpShape {
  u32 op_lo;        // first operand of the shape in the operand array
  u32 cnt;
  u16 start[5];     // operands are ordered by memory first: first local index of memory m; [4] = cnt
  u8 rank, sum;     // dimensions; sum of their logs
  u8 logs[8];       // log2 of the dimensions
  u8 tile_at[8];    // tile entries of dimension d start here in an operand's tile list
};

enum : u8 { DPO_CONTIG = 1, DPO_ROW_MAJOR = 2, DPO_COL_MAJOR = 4 };
struct DpOp {
  u32 moves_off, tile_off;
  u16 n_moves, n_actions;   // applicable Moves that fit the top limits; enumerated Moves
  u16 layout_id, rm_loc;    // equal ids = equal layouts; local index of the operand laid out row-major
  u32 cost;                 // move_cost of the operand
  u8 mem, vs, flags, pad;
};
struct DpMove {
  u32 imm, units;
  u16 rel, new_loc;         // position among the operand's enumerated Moves; the operand afterwards
  u8 mem, thr, miss, pad;   // destination; smallest limit code it fits; cache miss: no prologue / epilogue
};
// tile entry: local index of the tiled operand (in its own shape) | ok << 30 | applies << 31
enum : u32 { DPT_OK = 1u << 30, DPT_APPLIES = 1u << 31, DPT_LOC = 0xFFFFu };

struct DpFam {
  u8 kind, dtype, nd, nops;
  u8 logs[8];               // log2 of spec_shape
  u16 shape[3], move[3];    // per operand: its shape, and the Move family of that shape
  u16 accum, fill;          // Matmul: the accumulating family, the Fill of the output
  u32 child_off;            // child families: tiling dimension d to 2^e is entry child_at[d] + e
  u8 child_at[8];
  u32 base[10][4];          // first position of (level rank, memory of operand 0); Move and Fill use [.][0]
  u32 R[7], Q[7][4];        // three operands: positions of operands 1, 2 with level sum x; ... of memories below m1
};
// Goals: a product of operand lists (indices into the list array), or single Specs.
struct DpProduct { u32 fam; u32 list[3], n[3]; u32 first, count; };

constexpr u32 DP_NO_FAM = 0xFFFF;
inline u64 dp_pack(u32 fam, u32 i0, u32 i1, u32 i2) { return (u64)fam << 48 | (u64)i0 << 32 | (u64)i1 << 16 | i2; }

class OpTables {
 public:
  // Goal sets: every canonical Spec of a precompute, or a list of canonical Specs. Throws ModelError
  // when the job is outside what the factored form covers; the host planner then decides.
  void build_precompute(u32 size, Through through, const std::vector<Dtype>& dtypes);
  void build_goals(const std::vector<LogicalSpec>& goals);

  // Packed (family, operand indices) of a canonical Spec; false: not in these tables.
  bool locate(const LogicalSpec& ls, u64* out) const;
  // The same straight from a Spec blob; false also when the blob is not in canonical form.
  bool locate_blob(const u8* blob, size_t len, u64* out) const;
  LogicalSpec spec_of(u64 packed) const;

  std::vector<DpShape> shapes;
  std::vector<DpOp> ops;         // by shape, in key order
  std::vector<Aux> auxes;        // beside ops
  std::vector<DpMove> moves;
  std::vector<u32> tiles;
  std::vector<DpFam> fams;
  std::vector<u16> fam_child;
  std::vector<u32> stage_base;   // first position of every possible stage
  std::vector<u32> stage_key;    // kind << 16 | log-shape sum << 8 | level rank
  std::vector<DpProduct> products;
  std::vector<u16> lists;
  std::vector<u64> seeds;        // packed single goals
  u32 n_positions = 0;
  u32 max_records = 0;           // upper bound on a Spec's enumerated candidates
  u32 top_code[NMEM] = {0, 0, 0, 0};

 private:
  struct TmpOp {
    Aux aux;
    u32 shape, layout_id, rm;
    u32 moves_off, n_moves, n_actions, tile_off;
    u32 cost, units;
    u8 thr, flags;
    bool fits;
  };
  struct Dest { u32 lay, l1_lay; int to[4]; int vrf[2]; bool l1_ready; };   // layout ids; operands: -2 not worked out yet, -1 does not apply
  struct TmpShape {
    Shape s;
    std::vector<Dest> dests;
    std::vector<u32> ops;        // temporary ids
    std::vector<u32> child;      // shape after tiling dimension d to 2^e
    bool ready;
  };
  struct TmpMove { u32 imm, units, to; u16 rel; u8 mem, thr, miss; };
  u32 shape_id_(const Shape& s);
  u32 op_id_(u32 shape, const Aux& a) { return op_id_(shape, a.mem, a.vector_size, layout_id_(a.layout)); }
  u32 op_id_(u32 shape, Mem mem, u8 vs, u32 layout);
  u32 tiled_layouts_(u32 shape, u32 layout);
  u32 layout_id_(const Layout& l);
  u32 fam_id_(u8 kind, u8 dtype, const Shape& s);
  void close_operands_();
  void tabulate_op_(u32 o);
  int dest_op_(u32 shape, u32 d, Mem mem, int v);
  void finish_();
  void start_();
  u32 find_op_(u32 shape, u64 h, const u8* bytes, u32 len) const;

  Dtype dt_ = DT_U32;            // stands for every dtype of its size
  std::vector<TmpShape> tshapes_;
  std::vector<TmpOp> tops_;
  std::vector<TmpMove> tmoves_;
  std::vector<u32> ttiles_;      // temporary id | flags, as in tiles
  std::vector<Layout> layouts_;
  std::vector<u32> op_tab_, lay_tab_, fam_tab_, shape_tab_, tiled_tab_;   // open addressing, ids + 1
  std::vector<u64> tiled_keys_;                // shape << 32 | layout
  std::vector<u32> tiled_at_, tiled_;          // its entries: the layout after each tiling, as in ttiles_
  std::vector<u64> fam_keys_, shape_keys_;
  std::vector<u32> loc_;         // temporary id -> local index
  std::vector<u32> find_tab_;    // final: operand index + 1 by hash of (shape, key bytes)
  std::vector<std::vector<u32>> goal_lists_;   // precompute: temporary ids by shape
  std::vector<u64> fam_seed_;    // precompute: families whose full product is a goal set
};

}  // namespace mrl
