// Planning on the device (sm_100a): the closure of the goals, the ids and the candidate records
// of a fill, from the factored tables of optable.hpp.
//
// One cooperative launch; a Spec is handled by a warp, its enumerated candidates by the lanes.
//   closure   a bit per possible Spec in dense id order and a queue of those found; a round expands
//             what the round before queued
//   Specs     population counts and a scan turn bits into ids; per Spec a descriptor, the number of
//             its records and, after another scan, where they start
//   records   the candidates of a Spec, evaluated again with their children's ids, each written at
//             its place in the device's evaluation order (plan.cpp, cand_rank)
// The host planner (plan.cpp) builds the same arrays from tabulated Specs; the two agree byte for
// byte.
//
// What bounds it: latency of dependent table and bitmap reads that hit L1 and L2 (at size 8 in one dtype
// the tables are 1.0 MB and the bitmap another); the records, 32 bytes each, are the only large
// stream and are written once.
//
// Restates for the device: morello/src/target/cpu.rs:455-823 (action order),
// morello/src/scheduling/mod.rs:148-167 and the solvers cited in model/actions.hpp.
#include "devplan.hpp"
#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace mrl {
namespace {

struct SpecRef {
  const DpFam* f;
  u32 i[3];               // local operand indices
  u32 level;              // memory-level rank
};

struct Rec {
  u32 action, kind, nchild, imm, level, thr, peak, late, units;
  u64 child[3];           // packed family and operand indices
};

// Equal contiguous layouts on both sides of a Move become row-major.
__device__ __forceinline__ void canon_pair(const DpTables& t, const DpShape& s, u32& i0, u32& i1) {
  const DpOp &a = t.ops[s.op_lo + i0], &b = t.ops[s.op_lo + i1];
  if (a.layout_id == b.layout_id && (a.flags & DPO_CONTIG)) { i0 = a.rm_loc; i1 = b.rm_loc; }
}
__device__ __forceinline__ u64 pack_spec(u32 fam, u32 i0, u32 i1, u32 i2) { return (u64)fam << 48 | (u64)i0 << 32 | (u64)i1 << 16 | i2; }
__device__ __forceinline__ u64 move_spec(const DpTables& t, const DpShape& s, u32 fam, u32 i0, u32 i1) {
  canon_pair(t, s, i0, i1);
  return pack_spec(fam, i0, i1, 0);
}
__device__ __forceinline__ const DpOp& op_of(const DpTables& t, const SpecRef& s, int j) {
  return t.ops[t.shapes[s.f->shape[j]].op_lo + s.i[j]];
}
__device__ __forceinline__ u32 op_volume_log(const DpTables& t, const SpecRef& s, int j) { return t.shapes[s.f->shape[j]].sum; }

__device__ __forceinline__ SpecRef unpack_spec(const DpTables& t, u64 q) {
  SpecRef s;
  s.f = &t.fams[q >> 48];
  s.i[0] = (u32)(q >> 32) & 0xFFFFu;
  s.i[1] = (u32)(q >> 16) & 0xFFFFu;
  s.i[2] = (u32)q & 0xFFFFu;
  const u32 m0 = op_of(t, s, 0).mem;
  s.level = m0;
  if (s.f->nops == 2) s.level = max(m0, (u32)op_of(t, s, 1).mem);
  if (s.f->nops == 3) s.level = m0 + op_of(t, s, 1).mem + op_of(t, s, 2).mem;
  return s;
}

// Leaf kernels (model/actions.hpp, leaf_kernel_info), l-th of the Spec's kind.
__device__ bool leaf(const DpTables& t, const SpecRef& s, u32 l, u32& main, u32& level, u32& units) {
  const DpFam& f = *s.f;
  level = 0;
  units = 0;
  const DpOp& a = op_of(t, s, 0);
  if (f.kind == K_MOVE) {   // Assign
    if (l != 0) return false;
    const DpOp& b = op_of(t, s, 1);
    if (a.layout_id != b.layout_id) return false;
    if (op_volume_log(t, s, 0) == 0) {
      if ((a.mem != RF && a.mem != L1) || (b.mem != RF && b.mem != L1)) return false;
      main = a.cost + b.cost + 1;
      return true;
    }
    if (!(a.flags & DPO_CONTIG) || !(b.flags & DPO_CONTIG)) return false;
    const u32 vol = 1u << op_volume_log(t, s, 0);
    bool has_vrf = false;
    if (a.mem == VRF) { has_vrf = true; if (vol % a.vs != 0) return false; }
    if (b.mem == VRF) { has_vrf = true; if (vol % b.vs != 0) return false; }
    if (!has_vrf) return false;
    main = vol / (a.vs ? a.vs : b.vs);
    return true;
  }
  if (f.kind == K_FILL_ZERO) {
    if (l == 0) {           // MemsetZero
      main = 1;
      return a.mem != RF && a.mem != VRF && (a.flags & DPO_CONTIG);
    }
    if (l == 1) {           // ValueZero
      main = a.cost + 1;
      return op_volume_log(t, s, 0) == 0 && (a.mem == RF || a.mem == L1);
    }
    main = 1;               // VectorZero
    return (a.flags & DPO_CONTIG) && a.mem == VRF && a.vs != 0 && a.vs == (1u << op_volume_log(t, s, 0));
  }
  if (f.kind != K_MATMUL_ACCUM) return false;
  const DpOp &b = op_of(t, s, 1), &c = op_of(t, s, 2);
  if (l == 0) {             // MultAdd
    for (int j = 0; j < 3; j++) {
      const DpOp& o = op_of(t, s, j);
      if ((o.mem != RF && o.mem != L1) || op_volume_log(t, s, j) != 0) return false;
    }
    main = (f.dtype == DT_F32 ? 1u : (f.dtype == DT_BF16 ? 30u : 2u)) + a.cost + b.cost + c.cost;
    return true;
  }
  const DpShape &sa = t.shapes[f.shape[0]], &sb = t.shapes[f.shape[1]], &sc = t.shapes[f.shape[2]];
  if (l == 1) {             // BroadcastVecMultAdd
    if (f.dtype == DT_BF16) return false;
    if (c.mem != VRF || !(c.flags & DPO_CONTIG) || !(a.flags & DPO_CONTIG) || !(b.flags & DPO_CONTIG)) return false;
    if (sa.logs[0] != sc.logs[0] || sb.logs[0] != sc.logs[0]) return false;
    if (c.vs == 0 || (1u << sc.sum) % c.vs != 0) return false;
    bool hit = false;
    for (int side = 0; side < 2; side++) {
      const DpOp &x = side ? b : a, &y = side ? a : b;            // scalar, broadcast
      const DpShape &sx = side ? sb : sa, &sy = side ? sa : sb;
      if ((x.mem != RF && x.mem != L1) || y.mem != VRF || sx.sum != 0) continue;
      if (y.vs != c.vs || (1u << sy.sum) % c.vs != 0) continue;
      const u32 b1 = sy.logs[1], b2 = sy.logs[2], s1 = sx.logs[1], s2 = sx.logs[2], o1 = sc.logs[1], o2 = sc.logs[2];
      if (s1 == o1 && s2 == 0 && b1 == 0 && b2 == o2) hit = true;
      if (s1 == 0 && s2 == o2 && b1 == o1 && b2 == 0) hit = true;
    }
    if (!hit) return false;
    main = (1u << sc.sum) / c.vs * 2u + 1u;
    level = VRF;
    units = 1;
    return true;
  }
  if (f.dtype != DT_F32) return false;   // DotProductLoop
  if (sa.logs[0] != 0 || sa.logs[1] != 0 || sa.logs[2] < 3 || sc.sum != 0) return false;
  if (!(a.flags & DPO_ROW_MAJOR) || !(b.flags & DPO_COL_MAJOR) || !(a.flags & DPO_CONTIG) || !(b.flags & DPO_CONTIG)) return false;
  if ((a.vs != 0 && a.vs != 8) || (b.vs != 0 && b.vs != 8)) return false;
  if (!(a.mem == L1 || (a.mem == VRF && a.vs == 8))) return false;
  if (b.mem != L1 || (c.mem != RF && c.mem != L1)) return false;
  main = 8u * (1u << sa.logs[2]) / 32u + c.cost;
  level = VRF;
  units = 1;
  return true;
}

// What the enumeration of one Spec looks like: Moves of each operand, tile-outs, leaf kernels, tail.
struct EnumPlan {
  u32 end_move[3], end_tiles, end_leaf, end;   // enumeration indices
  u32 base_action[3], tile_action, leaf_action;
  u32 out_rank;
};
__device__ __forceinline__ EnumPlan enum_plan(const DpTables& t, const SpecRef& s) {
  EnumPlan p;
  const DpFam& f = *s.f;
  u32 e = 0, act = 0;
#pragma unroll
  for (int j = 0; j < 3; j++) {
    p.base_action[j] = act;
    if (j < f.nops) {
      const DpOp& o = op_of(t, s, j);
      e += o.n_moves;
      act += o.n_actions;
    }
    p.end_move[j] = e;
  }
  const DpShape& out = t.shapes[f.shape[f.nops - 1]];   // the output is every kind's last operand
  u32 ml = 0;
  for (u32 d = 0; d < out.rank; d++) ml = max(ml, (u32)out.logs[d]);
  p.out_rank = out.rank;
  p.tile_action = act;
  e += (ml + 1) * out.rank;
  act += (ml + 1) * out.rank;
  p.end_tiles = e;
  p.leaf_action = act;
  e += f.kind == K_MOVE ? 1u : (f.kind == K_MATMUL ? 0u : 3u);
  p.end_leaf = e;
  e += f.kind == K_MATMUL ? 1u : (f.kind == K_MATMUL_ACCUM ? (u32)f.logs[2] : 0u);
  p.end = e;
  return p;
}

// The e-th enumerated candidate; false when it does not apply. Children only if asked.
template <bool kChildren>
__device__ __forceinline__ bool record(const DpTables& t, const SpecRef& s, const EnumPlan& p, u32 e, Rec& r) {
  const DpFam& f = *s.f;
  r.level = r.thr = r.peak = r.late = r.units = 0;
  if (e < p.end_move[2]) {
    const int j = e < p.end_move[0] ? 0 : (e < p.end_move[1] ? 1 : 2);
    const u32 k = e - (j == 0 ? 0u : (j == 1 ? p.end_move[0] : p.end_move[1]));
    const u32 own = j == 0 ? s.i[0] : (j == 1 ? s.i[1] : s.i[2]);
    const DpOp& o = t.ops[t.shapes[f.shape[j]].op_lo + own];
    const DpMove mv = t.moves[o.moves_off + k];
    r.action = (j == 0 ? p.base_action[0] : (j == 1 ? p.base_action[1] : p.base_action[2])) + mv.rel;
    r.kind = MRL_CK_MOVE;
    r.imm = mv.imm;
    r.level = mv.mem;
    r.thr = mv.thr;
    r.units = mv.units;
    // operand directions (kind_direction): the last operand is written, the others are read; the accumulator is both
    const bool written = j == f.nops - 1, read = !written || f.kind == K_MATMUL_ACCUM;
    const bool pro = !mv.miss && read, epi = !mv.miss && written;
    r.nchild = 1u + pro + epi;
    if (f.kind == K_MOVE) {
      const u32 other = t.ops[t.shapes[f.shape[0]].op_lo + s.i[1 - j]].mem;
      r.late = max((u32)mv.mem, other) == s.level || ((pro || epi) && max((u32)mv.mem, (u32)o.mem) == s.level);
    } else {
      r.late = mv.mem == o.mem;
    }
    if (kChildren) {
      const u32 fam = (u32)(s.f - t.fams);
      const DpShape& own_shape = t.shapes[f.shape[j]];
      u32 b0 = j == 0 ? mv.new_loc : s.i[0], b1 = j == 1 ? mv.new_loc : s.i[1];
      const u32 b2 = j == 2 ? mv.new_loc : s.i[2];
      if (f.kind == K_MOVE) canon_pair(t, own_shape, b0, b1);
      const u64 body = pack_spec(fam, b0, b1, b2);
      const u64 prologue = pro ? move_spec(t, own_shape, f.move[j], own, mv.new_loc) : 0;
      const u64 epilogue = epi ? move_spec(t, own_shape, f.move[j], mv.new_loc, own) : 0;
      r.child[0] = pro ? prologue : body;
      r.child[1] = pro ? body : epilogue;
      r.child[2] = epilogue;   // read only if there are three
    }
    return true;
  }
  if (e < p.end_tiles) {
    const u32 q = e - p.end_move[2];
    const u32 se = q / p.out_rank, d = q - se * p.out_rank;   // tile size 2^se in output dimension d
    const DpShape& out = t.shapes[f.shape[f.nops - 1]];
    if (se >= out.logs[d]) return false;   // equal or larger
    const bool mm = f.nops == 3;
    const u32 sd = mm ? (d == 2 ? 3u : d) : d;                // the Spec dimension it tiles
    const u32 last = f.nops == 1 ? s.i[0] : (f.nops == 2 ? s.i[1] : s.i[2]);
    const u32 te = t.tiles[t.ops[out.op_lo + last].tile_off + out.tile_at[d] + se];
    if (!(te & DPT_APPLIES)) return false;
    bool ok = (te & DPT_OK) != 0;
    u32 n0 = s.i[0], n1 = s.i[1], n2 = s.i[2];
    if (f.nops == 1) n0 = te & DPT_LOC;
    else if (f.nops == 2) {
      n1 = te & DPT_LOC;
      const u32 x = t.tiles[t.ops[out.op_lo + s.i[0]].tile_off + out.tile_at[d] + se];   // both operands have the Spec's shape
      ok = ok && (x & DPT_OK);
      n0 = x & DPT_LOC;
    } else {
      n2 = te & DPT_LOC;
      if (d != 2) {   // batch, rows: also of the left operand
        const DpShape& s0 = t.shapes[f.shape[0]];
        const u32 x = t.tiles[t.ops[s0.op_lo + s.i[0]].tile_off + s0.tile_at[d] + se];
        ok = ok && (x & DPT_OK);
        n0 = x & DPT_LOC;
      }
      if (d != 1) {   // batch, columns: also of the right operand
        const DpShape& s1 = t.shapes[f.shape[1]];
        const u32 x = t.tiles[t.ops[s1.op_lo + s.i[1]].tile_off + s1.tile_at[d] + se];
        ok = ok && (x & DPT_OK);
        n1 = x & DPT_LOC;
      }
    }
    if (!ok) return false;
    r.action = p.tile_action + q;
    r.kind = MRL_CK_LOOP;
    r.nchild = 1;
    r.imm = 1u << (f.logs[sd] - se);
    if (kChildren) {
      const u32 cf = t.fam_child[f.child_off + f.child_at[sd] + se];
      if (f.kind == K_MOVE) canon_pair(t, t.shapes[t.fams[cf].shape[0]], n0, n1);
      r.child[0] = pack_spec(cf, n0, n1, n2);
    }
    return true;
  }
  // leaf kernels and the kind's tail are numbered by what applies before them
  u32 act = p.leaf_action;
  const u32 n_leaf = p.end_leaf - p.end_tiles, l = e - p.end_tiles;
  for (u32 k = 0; k < n_leaf; k++) {
    u32 main = 0, level = 0, units = 0;
    const bool hit = leaf(t, s, k, main, level, units);
    if (k == l) {
      if (!hit) return false;
      r.action = act;
      r.kind = MRL_CK_LEAF;
      r.nchild = 0;
      r.imm = main;
      r.level = level;
      r.units = units;
      r.thr = r.peak = units;   // registers: the code is the count
      return true;
    }
    act += hit;
  }
  if (f.kind == K_MATMUL) {   // ToAccum
    r.action = act;
    r.kind = MRL_CK_BLOCK;
    r.nchild = 2;
    r.imm = 0;
    if (kChildren) {
      r.child[0] = pack_spec(f.fill, s.i[2], 0, 0);
      r.child[1] = pack_spec(f.accum, s.i[0], s.i[1], s.i[2]);
    }
    return true;
  }
  // Split of the reduction dimension to 2^k
  const u32 k = e - p.end_leaf;
  const DpShape &s0 = t.shapes[f.shape[0]], &s1 = t.shapes[f.shape[1]];
  const u32* const t0 = t.tiles + t.ops[s0.op_lo + s.i[0]].tile_off + s0.tile_at[2];
  const u32* const t1 = t.tiles + t.ops[s1.op_lo + s.i[1]].tile_off + s1.tile_at[1];
  if (!(t0[k] & t1[k] & DPT_APPLIES)) return false;
  for (u32 q = 0; q < k; q++) act += (t0[q] & t1[q] & DPT_APPLIES) ? 1u : 0u;
  if (!(t0[k] & t1[k] & DPT_OK)) return false;
  r.action = act;
  r.kind = MRL_CK_LOOP;
  r.nchild = 1;
  r.imm = 1u << (f.logs[2] - k);
  if (kChildren) {
    r.child[0] = pack_spec(t.fam_child[f.child_off + f.child_at[2] + k], t0[k] & DPT_LOC, t1[k] & DPT_LOC, s.i[2]);
  }
  return true;
}

__device__ __forceinline__ u32 spec_pos(const DpTables& t, u64 q) {
  return dp_pos(t, t.fams[q >> 48], (u32)(q >> 32) & 0xFFFFu, (u32)(q >> 16) & 0xFFFFu, (u32)q & 0xFFFFu);
}

// Marks a Spec as existing and queues it for expansion when this is the first time. Every lane of
// the warp takes part (`have`: it brings a Spec); one queue slot request per warp. Most children
// exist already; an L1 copy of the word from before answers for those that it has.
__device__ __forceinline__ void add_specs(const PlanArgs& a, bool have, u64 q, u32 q_base, u32* q_count) {
  bool fresh = false;
  if (have) {
    const u32 pos = spec_pos(a.t, q);
    u32* const w = a.found + (pos >> 5);
    const u32 bit = 1u << (pos & 31u);
    if (!(*w & bit)) fresh = !(atomicOr(w, bit) & bit);
  }
  const u32 who = __ballot_sync(0xFFFFFFFFu, fresh);
  if (!who) return;
  const u32 lane = threadIdx.x & 31u, leader = __ffs(who) - 1;
  u32 at = 0;
  if (lane == leader) at = atomicAdd(q_count, __popc(who));
  at = __shfl_sync(0xFFFFFFFFu, at, leader);
  if (fresh) a.queue[q_base + at + __popc(who & ((1u << lane) - 1u))] = q;
}

__device__ __forceinline__ void seed_goals(const PlanArgs& a, u32 gtid, u32 gthreads, u32* q_count) {
  for (u32 k0 = gtid & ~31u; k0 < a.n_seeds; k0 += gthreads) {
    const u32 k = k0 + (threadIdx.x & 31u);
    add_specs(a, k < a.n_seeds, k < a.n_seeds ? a.seeds[k] : 0ull, 0, q_count);
  }
  for (u32 b = blockIdx.x; b < a.n_products; b += gridDim.x) {
    const DpProduct p = a.products[b];
    const DpFam& f = a.t.fams[p.fam];
    for (u32 k0 = threadIdx.x & ~31u; k0 < p.count; k0 += kPlanBlock) {
      const u32 k = k0 + (threadIdx.x & 31u);
      bool have = k < p.count;
      u64 q = 0;
      if (have) {
        u32 rest = p.first + k;
        const u32 i2 = f.nops > 2 ? a.lists[p.list[2] + rest % p.n[2]] : 0u;
        rest /= p.n[2];
        const u32 i1 = f.nops > 1 ? a.lists[p.list[1] + rest % p.n[1]] : 0u;
        rest /= p.n[1];
        const u32 i0 = a.lists[p.list[0] + rest];
        if (f.kind == K_MOVE) {   // not canonical: equal contiguous layouts other than row-major
          const DpShape& s = a.t.shapes[f.shape[0]];
          const DpOp &x = a.t.ops[s.op_lo + i0], &y = a.t.ops[s.op_lo + i1];
          if (x.layout_id == y.layout_id && (x.flags & DPO_CONTIG) && !(x.flags & DPO_ROW_MAJOR)) have = false;
        }
        q = pack_spec(p.fam, i0, i1, i2);
      }
      add_specs(a, have, q, 0, q_count);
    }
  }
}

// One closure round: the children of the Specs queued by the round before.
__device__ __forceinline__ void closure_round(const PlanArgs& a, u32 q_lo, u32 q_hi, u32 gwarp, u32 gwarps, u32* q_count) {
  const u32 lane = threadIdx.x & 31u;
  for (u32 k = q_lo + gwarp; k < q_hi; k += gwarps) {
    const SpecRef s = unpack_spec(a.t, __ldcg(a.queue + k));
    const EnumPlan p = enum_plan(a.t, s);
    for (u32 e0 = 0; e0 < p.end; e0 += 32) {
      Rec r;
      r.nchild = 0;
      if (!(e0 + lane < p.end && record<true>(a.t, s, p, e0 + lane, r))) r.nchild = 0;
#pragma unroll
      for (u32 j = 0; j < 3; j++)
        if (__any_sync(0xFFFFFFFFu, j < r.nchild)) add_specs(a, j < r.nchild, r.child[j], q_hi, q_count);
    }
  }
}

__device__ __forceinline__ unsigned long long block_sum(unsigned long long v) {
  __shared__ unsigned long long part[kPlanBlock / 32];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
  __syncthreads();
  unsigned long long s = 0;
  for (int k = 0; k < kPlanBlock / 32; k++) s += part[k];
  return s;
}
__device__ __forceinline__ u32 block_excl(u32 v, u32* total) {
  __shared__ u32 part[kPlanBlock / 32];
  const u32 lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
  u32 inc = v;
  for (int o = 1; o < 32; o <<= 1) {
    const u32 x = __shfl_up_sync(0xFFFFFFFFu, inc, o);
    if (lane >= (u32)o) inc += x;
  }
  __syncthreads();
  if (lane == 31) part[w] = inc;
  __syncthreads();
  u32 before = 0, all = 0;
  for (u32 k = 0; k < kPlanBlock / 32; k++) {
    if (k < w) before += part[k];
    all += part[k];
  }
  *total = all;
  return before + inc - v;
}
// The part of [0, n) a block scans: whole tiles of kPlanBlock, evenly.
__device__ __forceinline__ void block_range(u32 n, u32& lo, u32& hi) {
  const u32 tiles = (n + kPlanBlock - 1) / kPlanBlock, per = (tiles + gridDim.x - 1) / gridDim.x;
  lo = min(n, blockIdx.x * per * kPlanBlock);
  hi = min((unsigned long long)n, (unsigned long long)lo + (unsigned long long)per * kPlanBlock);
}
__device__ __forceinline__ unsigned long long sums_before(const unsigned long long* sums) {
  unsigned long long v = 0;
  for (u32 k = threadIdx.x; k < blockIdx.x; k += kPlanBlock) v += sums[k];
  return block_sum(v);
}

__global__ void __launch_bounds__(kPlanBlock) plan_kernel(const __grid_constant__ PlanArgs a) {
  cg::grid_group grid = cg::this_grid();
  const u32 gtid = blockIdx.x * kPlanBlock + threadIdx.x, gthreads = gridDim.x * kPlanBlock;
  const u32 lane = threadIdx.x & 31u;
  const u32 gwarp = gtid >> 5, gwarps = gthreads >> 5;
  PlanCtl* const ctl = a.ctl;

  if (a.phases & DPP_CLOSURE) {
    // Four counters in turn: one counts what this round queues, one was read behind the last
    // barrier, one is cleared for the round after next.
    seed_goals(a, gtid, gthreads, &ctl->queued[0]);
    grid.sync();
    u32 q_lo = 0, q_hi = __ldcg(&ctl->queued[0]), round = 0;
    if (gtid == 0) ctl->n_goals = q_hi;
    while (q_hi > q_lo) {
      round++;
      if (gtid == 0) ctl->queued[(round + 2) & 3] = 0;
      closure_round(a, q_lo, q_hi, gwarp, gwarps, &ctl->queued[round & 3]);
      grid.sync();
      q_lo = q_hi;
      q_hi += __ldcg(&ctl->queued[round & 3]);
    }
    if (gtid == 0) ctl->rounds = round;
    // bits to ids
    u32 lo, hi;
    block_range(a.n_words, lo, hi);
    unsigned long long own = 0;
    for (u32 w = lo + threadIdx.x; w < hi; w += kPlanBlock) own += __popc(__ldcg(a.found + w));
    own = block_sum(own);
    if (threadIdx.x == 0) a.block_sums[blockIdx.x] = own;
    grid.sync();
    u32 carry = (u32)sums_before(a.block_sums);
    for (u32 w0 = lo; w0 < hi; w0 += kPlanBlock) {
      const u32 w = w0 + threadIdx.x;
      const u32 word = w < hi ? __ldcg(a.found + w) : 0u;
      u32 total;
      const u32 ex = block_excl(__popc(word), &total);
      if (w < hi) a.rank[w] = make_uint2(word, carry + ex);
      carry += total;
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {   // the last block's range ends at the last word
      ctl->n_specs = carry;
      a.stage_lo[a.n_stages] = carry;
    }
    grid.sync();
    for (u32 g = gtid; g < a.n_stages; g += gthreads) {
      const uint2 w = __ldcg(a.rank + (a.stage_base[g] >> 5));
      a.stage_lo[g] = w.y + __popc(w.x & ((1u << (a.stage_base[g] & 31u)) - 1u));
    }
  }

  if (a.phases & DPP_SPECS) {
    const u32 n = __ldcg(&ctl->n_specs);
    if (n > a.cap_specs) return;   // uniform: the caller enlarges and launches again
    for (u32 k = gwarp; k < n; k += gwarps) {
      const u64 q = __ldcg(a.queue + k);
      const SpecRef s = unpack_spec(a.t, q);
      const EnumPlan p = enum_plan(a.t, s);
      u32 count = 0;
      for (u32 e0 = 0; e0 < p.end; e0 += 32) {
        Rec r;
        const bool hit = e0 + lane < p.end && record<false>(a.t, s, p, e0 + lane, r);
        count += __popc(__ballot_sync(0xFFFFFFFFu, hit));
      }
      if (lane == 0) {
        const u32 id = dp_id(a.t, spec_pos(a.t, q));
        uint4* const h = reinterpret_cast<uint4*>(a.hdrs + id);
        h[0] = make_uint4(0, 0, 0, 0);
        h[1] = make_uint4(0, 0, 0, count);
        a.desc[id] = q;
      }
    }
    grid.sync();
    u32 lo, hi;
    block_range(n, lo, hi);
    unsigned long long own = 0;
    for (u32 i = lo + threadIdx.x; i < hi; i += kPlanBlock) own += a.hdrs[i].ncand;
    own = block_sum(own);
    if (threadIdx.x == 0) a.block_sums[blockIdx.x] = own;
    grid.sync();
    unsigned long long carry = sums_before(a.block_sums);
    for (u32 i0 = lo; i0 < hi; i0 += kPlanBlock) {
      const u32 i = i0 + threadIdx.x;
      u32 total;
      const u32 ex = block_excl(i < hi ? a.hdrs[i].ncand : 0u, &total);
      if (i < hi) a.hdrs[i].cand_off = (u32)(carry + ex);   // the total is checked to fit 32 bits
      carry += total;
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) ctl->n_cands = carry;
    grid.sync();
  }

  if (a.phases & DPP_RECORDS) {
    const u32 n = __ldcg(&ctl->n_specs);
    if (n > a.cap_specs || __ldcg(&ctl->n_cands) > a.cap_cands) return;
    __shared__ u64 keys_all[kPlanBlock / 32][DP_MAX_RECORDS];
    u64* const keys = keys_all[threadIdx.x >> 5];
    for (u32 id = gwarp; id < n; id += gwarps) {
      const SpecRef s = unpack_spec(a.t, a.desc[id]);
      const u32 off = a.hdrs[id].cand_off;
      const EnumPlan p = enum_plan(a.t, s);
      // evaluation order: cand_rank, then the action number (numbers are unique and ascend with the enumeration)
      u32 count = 0;
      __syncwarp();
      for (u32 e0 = 0; e0 < p.end; e0 += 32) {
        Rec r;
        const bool hit = e0 + lane < p.end && record<false>(a.t, s, p, e0 + lane, r);
        const u32 hits = __ballot_sync(0xFFFFFFFFu, hit);
        if (hit) {
          u64 key;
          if (r.late) key = (u64(1) << 40) | (0xFFFFFFFFu - r.imm);
          else key = (u64)(r.kind == MRL_CK_LEAF ? 0 : (r.kind == MRL_CK_LOOP ? 1 : (r.kind == MRL_CK_BLOCK ? 2 : 3))) << 32 |
                     (r.kind == MRL_CK_MOVE ? r.imm : 0u);
          keys[count + __popc(hits & ((1u << lane) - 1u))] = key << 16 | r.action;
        }
        count += __popc(hits);
      }
      __syncwarp();
      u32 seen = 0;
      for (u32 e0 = 0; e0 < p.end; e0 += 32) {
        Rec r;
        const bool hit = e0 + lane < p.end && record<true>(a.t, s, p, e0 + lane, r);
        const u32 hits = __ballot_sync(0xFFFFFFFFu, hit);
        const u32 me = seen + __popc(hits & ((1u << lane) - 1u));
        seen += __popc(hits);
        if (!hit) continue;
        const u64 key = keys[me];
        u32 at = 0;
        for (u32 k = 0; k < count; k++) at += keys[k] < key;
        u32 c0 = 0, c1 = 0, c2 = 0;
        if (r.nchild > 0) c0 = dp_id(a.t, spec_pos(a.t, r.child[0]));
        if (r.nchild > 1) c1 = dp_id(a.t, spec_pos(a.t, r.child[1]));
        if (r.nchild > 2) c2 = dp_id(a.t, spec_pos(a.t, r.child[2]));
        uint4* const out = reinterpret_cast<uint4*>(a.cands + off + at);
        out[0] = make_uint4(r.action | r.kind << 16 | r.nchild << 24, r.imm, r.level | r.thr << 8 | r.peak << 16 | r.late << 24, r.units);
        out[1] = make_uint4(c0, c1, c2, 0);
      }
    }
  }
}

}  // namespace

int plan_kernel_blocks_per_sm() {
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, plan_kernel, kPlanBlock, 0) != cudaSuccess) return 0;
  return n;
}

cudaError_t launch_plan_kernel(const PlanArgs& a, int blocks, cudaStream_t stream) {
  void* args[] = {const_cast<PlanArgs*>(&a)};
  return cudaLaunchCooperativeKernel((const void*)plan_kernel, dim3(blocks), dim3(kPlanBlock), args, 0, stream);
}

}  // namespace mrl
