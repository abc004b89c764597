// Arithmetic on the factored planning tables (optable.hpp) that device code shares: where a Spec
// lies in the dense id order, and its id.
#pragma once
#include "optable.hpp"
#include <cuda_runtime.h>

namespace mrl {

struct DpTables {   // device copies
  const DpShape* shapes;
  const DpOp* ops;
  const DpMove* moves;
  const u32* tiles;
  const DpFam* fams;
  const u16* fam_child;
  const uint2* rank;   // per 32 positions: which exist, and how many exist before them
};

// Position of a Spec given by family and local operand indices (optable.hpp: level rank, then
// operand order inside it).
__device__ __forceinline__ u32 dp_pos_move(const DpTables& t, const DpFam& f, u32 i0, u32 i1) {
  const DpShape& s = t.shapes[f.shape[0]];
  const u32 m0 = t.ops[s.op_lo + i0].mem, m1 = t.ops[s.op_lo + i1].mem, L = max(m0, m1);
  const u32 lo = s.start[L], hi = s.start[L + 1], c = hi - lo;
  if (m0 < L) return f.base[L][0] + i0 * c + (i1 - lo);
  return f.base[L][0] + lo * c + (i0 - lo) * hi + i1;
}
__device__ __forceinline__ u32 dp_pos_fill(const DpTables& t, const DpFam& f, u32 i0) {
  const DpShape& s = t.shapes[f.shape[0]];
  const u32 m0 = t.ops[s.op_lo + i0].mem;
  return f.base[m0][0] + i0 - s.start[m0];
}
__device__ __forceinline__ u32 dp_pos_matmul(const DpTables& t, const DpFam& f, u32 i0, u32 i1, u32 i2) {
  const DpShape &s0 = t.shapes[f.shape[0]], &s1 = t.shapes[f.shape[1]], &s2 = t.shapes[f.shape[2]];
  const u32 m0 = t.ops[s0.op_lo + i0].mem, m1 = t.ops[s1.op_lo + i1].mem, m2 = t.ops[s2.op_lo + i2].mem;
  const u32 x = m1 + m2;
  return f.base[m0 + x][m0] + (i0 - s0.start[m0]) * f.R[x] + f.Q[x][m1] + (i1 - s1.start[m1]) * (u32)(s2.start[m2 + 1] - s2.start[m2]) +
         (i2 - s2.start[m2]);
}
__device__ __forceinline__ u32 dp_pos(const DpTables& t, const DpFam& f, u32 i0, u32 i1, u32 i2) {
  if (f.nops == 3) return dp_pos_matmul(t, f, i0, i1, i2);
  return f.nops == 2 ? dp_pos_move(t, f, i0, i1) : dp_pos_fill(t, f, i0);
}
__device__ __forceinline__ u32 dp_id(const DpTables& t, u32 pos) {
  const uint2 w = t.rank[pos >> 5];
  return w.y + __popc(w.x & ((1u << (pos & 31u)) - 1u));
}

}  // namespace mrl
