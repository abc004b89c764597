// Text form of a reconstructed implementation: one line per node of the tree that results from
// re-applying, from a goal Spec down, the action the database stores for each (Spec, limits)
// (the walk of morello/src/reconstruct.rs:14-80 and FilesDatabase::get_impl,
// morello/src/db/mod.rs:505-516). The layout of a line is this library's own; the reference's
// pretty printer (morello/src/pprint.rs) prints tensors and loops of the generated code, which is
// outside the path built here.
//
//   <2 spaces per level><Spec> @ [rf, vrf, l1, gl]: #<action> <what> cost <main> peaks [..] depth <d>
#pragma once
#include "actions.hpp"

namespace mrl {

inline const char* leaf_kernel_name(u8 k) {
  static const char* n[] = {"MultAdd", "BroadcastVecMultAdd", "DotProductLoop", "Assign", "MemsetZero", "ValueZero", "VectorZero"};
  return k < 7 ? n[k] : "?";
}

inline std::string action_text(const Candidate& c) {
  switch (c.what) {
    case ACT_MOVE: {
      std::string s = "Move(operand " + std::to_string(c.arg0) + " -> " + mem_name((Mem)c.arg1);
      if (mem_has_layout((Mem)c.arg1)) s += ", layout " + c.lay.str();
      if (c.arg2) s += ", vector " + std::to_string(c.arg2);
      return s + ")";
    }
    case ACT_TILE_OUT: return "TileOut(dim " + std::to_string(c.arg0) + ", size " + std::to_string(c.arg2) + ")";
    case ACT_SPLIT: return "Split(k " + std::to_string(c.arg2) + ")";
    case ACT_KERNEL: return std::string("Kernel(") + leaf_kernel_name(c.arg0) + ")";
    default: return "ToAccum";
  }
}

// The action with a given number, as text needs it (what, operand or dimension, destination or size):
// found by the enumeration's counts (tabulate_candidates), without working out any other action.
// False: the Spec has no such action.
inline bool action_of(const LogicalSpec& spec, u32 action, Candidate& c) {
  c.action = (u16)action;
  u32 at = 0;
  for (int i = 0; i < spec.nops(); i++) {
    const TensorSpec op = spec.operand(i);
    bool contains_source = false;
    auto take = [&](Mem mem, const Layout& layout, u32 vs) {
      if (at++ != action) return false;
      c.what = ACT_MOVE;
      c.kind = CK_MOVE;
      c.arg0 = (u8)i;
      c.arg1 = (u8)mem;
      c.arg2 = vs;
      c.lay = layout;
      return true;
    };
    const std::vector<Mem> mems = possible_destination_memories(op.aux.mem);
    for (const Layout& layout : move_destination_layouts(op.shape, op.dtype)) {
      contains_source = contains_source || layout == op.aux.layout;
      for (Mem mem : mems) {
        const std::vector<u32>& vb = mem_vector_bytes(mem);
        if (vb.empty()) { if (take(mem, layout, 0)) return true; }
        else for (u32 b : vb) if (take(mem, layout, b / dtype_size(op.dtype))) return true;
      }
    }
    if (!contains_source)
      for (Mem mem : mems)
        if (!mem_is_addressed(mem) && take(mem, op.aux.layout, 0)) return true;
  }
  const Shape out = spec.operand_shape(kind_output_index(spec.kind));
  u32 max_dim = 0;
  for (int d = 0; d < out.n; d++) if (out[d] > max_dim) max_dim = out[d];
  for (u32 size : dim_range_pow2(max_dim, true))
    for (int dim = 0; dim < out.n; dim++)
      if (at++ == action) {
        c.what = ACT_TILE_OUT;
        c.kind = CK_LOOP;
        c.arg0 = (u8)dim;
        c.arg2 = size;
        return true;
      }
  std::vector<Candidate> leaves;
  at = tabulate_leaves(spec, at, leaves);
  for (const Candidate& l : leaves) if (l.action == action) { c = l; return true; }
  if (spec.kind == K_MATMUL && at == action) {
    c.what = ACT_TO_ACCUM;
    c.kind = CK_BLOCK;
    return true;
  }
  if (spec.kind == K_MATMUL_ACCUM) {
    const TensorSpec a = spec.operand(0), b = spec.operand(1);
    const u32 bt = spec.spec_shape[0], m = spec.spec_shape[1], n = spec.spec_shape[3];
    for (u32 k : dim_range_pow2(spec.spec_shape[2], false)) {
      if (!tensorspec_valid_tile_shape(a, Shape{bt, m, k}) || !tensorspec_valid_tile_shape(b, Shape{bt, k, n})) continue;
      if (at++ == action) {
        c.what = ACT_SPLIT;
        c.kind = CK_LOOP;
        c.arg2 = k;
        return true;
      }
    }
  }
  return false;
}

inline std::string limits_text(const u64 v[NMEM]) {
  std::string s = "[";
  for (int i = 0; i < NMEM; i++) { if (i) s += ", "; s += std::to_string(v[i]); }
  return s + "]";
}

inline std::string impl_line(int level, const LogicalSpec& spec, const u64 limits[NMEM], u32 action, const std::string& what,
                             u32 main, const u64 peaks[NMEM], u32 depth) {
  return std::string((size_t)level * 2, ' ') + spec.str() + " @ " + limits_text(limits) + ": #" + std::to_string(action) + " " +
         what + " cost " + std::to_string(main) + " peaks " + limits_text(peaks) + " depth " + std::to_string(depth) + "\n";
}

}  // namespace mrl
