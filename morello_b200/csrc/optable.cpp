// Interned operands and their Moves and tiles: the host half of planning on the device. See optable.hpp.
#include "optable.hpp"
#include <algorithm>

namespace mrl {

namespace {

u64 mix(u64 h, u64 w) {
  h = (h ^ w) * 0xD6E8FEB86659FD93ull;
  return h ^ (h >> 32);
}
u64 layout_hash(const Layout& l) {
  u64 h = mix(0x9E3779B97F4A7C15ull, (u64)l.n << 8 | l.contig);
  for (int i = 0; i < l.n; i++) h = mix(h, (u64)l.d[i].ldim << 24 | (u64)l.d[i].kind << 16 | l.d[i].size);
  return h ^ (h >> 29);
}
// An operand's bytes in a Spec key (LogicalSpec::key_into).
int aux_bytes(const Aux& a, u8* s) {
  int p = 0;
  s[p++] = (u8)a.mem; s[p++] = a.vector_size; s[p++] = a.layout.n; s[p++] = a.layout.contig;
  for (int j = 0; j < a.layout.n; j++) {
    s[p++] = a.layout.d[j].ldim; s[p++] = a.layout.d[j].kind;
    s[p++] = (u8)(a.layout.d[j].size & 0xff); s[p++] = (u8)(a.layout.d[j].size >> 8);
  }
  return p;
}
u64 bytes_hash(u32 shape, const u8* s, u32 len) {
  u64 h = mix(0x9E3779B97F4A7C15ull, (u64)shape << 32 | len);
  for (u32 i = 0; i < len; i += 4) { u32 w; memcpy(&w, s + i, 4); h = mix(h, w); }   // operand encodings are multiples of 4 bytes
  return h ^ (h >> 29);
}
int log2_of(u32 d) { return 31 - __builtin_clz(d); }
u64 dims_key(const Shape& s) {
  u64 k = s.n;
  for (int i = 0; i < s.n; i++) {
    if (!is_pow2(s[i]) || s[i] > (1u << 15)) throw ModelError("dimensions outside the factored planner's range");
    k |= (u64)log2_of(s[i]) << (4 + 4 * i);
  }
  return k;
}
// Lookup-or-insert position in an open-addressing table of ids + 1, kept at most half full.
template <class Eq, class HashOf>
size_t probe(std::vector<u32>& tab, size_t count, u64 h, Eq eq, HashOf hash_of) {
  if ((count + 1) * 2 > tab.size()) {
    std::vector<u32> bigger(std::max<size_t>(64, tab.size() * 4), 0);
    for (u32 v : tab)
      if (v) {
        size_t i = hash_of(v - 1) & (bigger.size() - 1);
        while (bigger[i]) i = (i + 1) & (bigger.size() - 1);
        bigger[i] = v;
      }
    tab.swap(bigger);
  }
  size_t i = h & (tab.size() - 1);
  while (tab[i] && !eq(tab[i] - 1)) i = (i + 1) & (tab.size() - 1);
  return i;
}
u64 fam_key(u8 kind, u8 dtype, const Shape& s) { return dims_key(s) | (u64)kind << 40 | (u64)dtype << 44; }

u32 code_of_units(int mem, u64 units) {   // smallest limit code whose value is at least `units` (plan.cpp, code_ceil)
  return mem_counts_registers((Mem)mem) ? (u32)units : bit_length(next_binary_power(units));
}

}  // namespace

u32 OpTables::shape_id_(const Shape& s) {
  const u64 key = dims_key(s);
  const size_t at = probe(shape_tab_, tshapes_.size(), mix(1, key), [&](u32 i) { return shape_keys_[i] == key; },
                          [&](u32 i) { return mix(1, shape_keys_[i]); });
  if (shape_tab_[at]) return shape_tab_[at] - 1;
  const u32 id = (u32)tshapes_.size();
  shape_tab_[at] = id + 1;
  shape_keys_.push_back(key);
  tshapes_.emplace_back();
  tshapes_[id].s = s;
  tshapes_[id].ready = false;
  std::vector<u32> child;
  for (int d = 0; d < s.n; d++)
    for (u32 e = 1; e < s[d]; e *= 2) {
      Shape t = s;
      t[d] = e;
      child.push_back(shape_id_(t));
    }
  tshapes_[id].child.swap(child);
  return id;
}

u32 OpTables::layout_id_(const Layout& l) {
  const size_t at = probe(lay_tab_, layouts_.size(), layout_hash(l), [&](u32 i) { return layouts_[i] == l; },
                          [&](u32 i) { return layout_hash(layouts_[i]); });
  if (lay_tab_[at]) return lay_tab_[at] - 1;
  layouts_.push_back(l);
  lay_tab_[at] = (u32)layouts_.size();
  return (u32)layouts_.size() - 1;
}

u32 OpTables::op_id_(u32 shape, Mem mem, u8 vs, u32 layout) {
  auto hash = [](u32 sh, u32 m, u32 v, u32 l) { return mix(mix(3, (u64)sh << 32 | l), (u64)m << 8 | v); };
  const size_t at = probe(op_tab_, tops_.size(), hash(shape, mem, vs, layout),
                          [&](u32 i) { const TmpOp& t = tops_[i]; return t.shape == shape && t.layout_id == layout && t.aux.mem == mem && t.aux.vector_size == vs; },
                          [&](u32 i) { const TmpOp& t = tops_[i]; return hash(t.shape, t.aux.mem, t.aux.vector_size, t.layout_id); });
  if (op_tab_[at]) return op_tab_[at] - 1;
  const u32 id = (u32)tops_.size();
  op_tab_[at] = id + 1;
  tops_.emplace_back();
  TmpOp& t = tops_[id];
  t.aux.mem = mem;
  t.aux.vector_size = vs;
  t.aux.layout = layouts_[layout];
  t.shape = shape;
  t.layout_id = layout;
  TensorSpec ts;
  ts.shape = tshapes_[shape].s;
  ts.dtype = dt_;
  ts.aux = t.aux;
  t.cost = move_cost(ts);
  const u64 units = tensorspec_memory_units(ts);
  t.units = (u32)units;
  const u32 thr = code_of_units(mem, (u32)units);
  t.fits = thr <= top_code[mem];
  t.thr = t.fits ? (u8)thr : 0;
  t.flags = (t.aux.layout.fully_contiguous() ? DPO_CONTIG : 0) | (t.aux.layout.is_row_major() ? DPO_ROW_MAJOR : 0) |
            (t.aux.layout.is_col_major() ? DPO_COL_MAJOR : 0);
  tshapes_[shape].ops.push_back(id);
  return id;
}

// The operand a Move to destination layout d of the shape ends as (plan_move, the cases whose
// result does not depend on the moved operand): v = vector width index for VRF.
int OpTables::dest_op_(u32 shape, u32 d, Mem mem, int v) {
  Dest& e = tshapes_[shape].dests[d];
  int& slot = mem == VRF ? e.vrf[v] : e.to[mem];
  if (slot != -2) return slot;
  TensorSpec t;
  t.shape = tshapes_[shape].s;
  t.dtype = dt_;
  t.aux.mem = mem;
  t.aux.vector_size = mem == VRF ? (u8)(mem_vector_bytes(VRF)[v] / dtype_size(dt_)) : 0;
  if (mem_has_layout(mem)) {
    t.aux.layout = layouts_[mem == L1 ? e.l1_lay : e.lay];
    t.aux.layout.contig = t.aux.layout.n;
  }
  int to = -1;
  if (tensorspec_canonicalize(t) == CANON_OK) to = (int)op_id_(shape, t.aux);   // no new shape: `slot` stays where it is
  slot = to;
  return to;
}

// What tiling does to a layout (tile_operand, the part that an operand's memory has no say in), for
// every dimension and tile size of the shape: layout id | DPT_OK | DPT_APPLIES. Operands in several
// memories share layouts, so this is worked out once per shape and layout: it is most of the cost of
// an operand.
u32 OpTables::tiled_layouts_(u32 shape, u32 layout) {
  const u64 key = (u64)shape << 32 | layout;
  const size_t at = probe(tiled_tab_, tiled_keys_.size(), mix(4, key), [&](u32 i) { return tiled_keys_[i] == key; },
                          [&](u32 i) { return mix(4, tiled_keys_[i]); });
  if (tiled_tab_[at]) return tiled_at_[tiled_tab_[at] - 1];
  tiled_keys_.push_back(key);
  tiled_at_.push_back((u32)tiled_.size());
  tiled_tab_[at] = (u32)tiled_keys_.size();
  const Shape s = tshapes_[shape].s;
  const Layout own = layouts_[layout];
  Layout nl, canon;
  for (int d = 0; d < s.n; d++)
    for (u32 e = 1; e < s[d]; e *= 2) {
      Shape tile = s;
      tile[d] = e;
      u32 entry = 0;
      if (layout_update_for_tiling(own, s, tile, nl)) {
        entry = DPT_APPLIES;
        if (layout_update_for_tiling(nl, tile, tile, canon)) {
          const u32 id = layout_id_(canon);
          if (id > 0x3FFFFFFFu) throw ModelError("too many layouts");
          entry |= DPT_OK | id;
        }
      }
      tiled_.push_back(entry);
    }
  if (!layout_update_for_tiling(own, s, s, nl) || nl != own) throw ModelError("an operand is not canonical");
  return tiled_at_.back();
}

// Moves and tiles of one operand (operand_moves and tile_operand of model/actions.hpp, with what
// they share between operands of one shape worked out once).
void OpTables::tabulate_op_(u32 o) {
  const u32 sh = tops_[o].shape;
  const Mem mem = tops_[o].aux.mem;
  const u8 vs = tops_[o].aux.vector_size;
  const u32 lay = tops_[o].layout_id;
  const bool contig = (tops_[o].flags & DPO_CONTIG) != 0;
  const Shape shape = tshapes_[sh].s;
  if (!tshapes_[sh].ready) {
    for (const Layout& l : move_destination_layouts(shape, dt_)) {
      Dest e;
      e.lay = layout_id_(l);
      e.l1_lay = 0;
      e.l1_ready = false;
      for (int& x : e.to) x = -2;
      for (int& x : e.vrf) x = -2;
      tshapes_[sh].dests.push_back(e);
    }
    tshapes_[sh].ready = true;
  }
  const u32 src_cost = tops_[o].cost;
  u32 n_actions = 0;
  const u32 moves_off = (u32)tmoves_.size();
  auto emit = [&](int to, bool miss) {
    const u32 rel = n_actions++;
    if (to < 0 || (u32)to == o || !tops_[to].fits) return;
    const TmpOp& t = tops_[to];
    tmoves_.push_back(TmpMove{src_cost + t.cost, t.units, (u32)to, (u16)rel, (u8)t.aux.mem, t.thr, (u8)miss});
  };
  auto same_layout_in_l1 = [&]() { return (int)op_id_(sh, L1, 0, lay); };
  bool contains_source = false;
  const size_t n_dests = tshapes_[sh].dests.size();
  const bool from_l1 = mem == L1, from_gl = mem == GL;
  for (u32 d = 0; d < n_dests; d++) {
    contains_source |= tshapes_[sh].dests[d].lay == lay;
    // possible_destination_memories, in its order
    if (mem == RF) emit(dest_op_(sh, d, RF, 0), false);
    if (from_gl) emit(dest_op_(sh, d, GL, 0), false);
    if (from_l1 || from_gl) {
      if (!tshapes_[sh].dests[d].l1_ready) {
        Layout l1;
        if (!layout_canonicalize(layouts_[tshapes_[sh].dests[d].lay], shape, l1)) throw ModelError("destination layout does not apply to the moved tensor");
        const u32 id = layout_id_(l1);
        tshapes_[sh].dests[d].l1_lay = id;
        tshapes_[sh].dests[d].l1_ready = true;
      }
      const bool miss = tshapes_[sh].dests[d].l1_lay == lay;
      emit(miss ? same_layout_in_l1() : dest_op_(sh, d, L1, 0), miss);
    }
    if (from_l1) emit(dest_op_(sh, d, RF, 0), false);
    if (from_l1 || mem == VRF)
      for (int v = 0; v < 2; v++) emit(dest_op_(sh, d, VRF, v), false);
  }
  if (!contains_source && (from_l1 || from_gl)) {
    Layout l;
    if (!layout_canonicalize(layouts_[lay], shape, l)) throw ModelError("destination layout does not apply to the moved tensor");
    if (l != layouts_[lay]) throw ModelError("an operand's layout is not canonical");
    emit(same_layout_in_l1(), true);
  }
  TmpOp& t = tops_[o];
  t.moves_off = moves_off;
  t.n_moves = (u32)tmoves_.size() - moves_off;
  t.n_actions = n_actions;
  // row-major in the same memory: what the matching-layouts rule of Move Specs turns the operand into
  u32 rm = o;
  if (mem_has_layout(mem) && contig) rm = op_id_(sh, mem, vs, layout_id_(layout_row_major(shape)));
  tops_[o].rm = rm;
  // tiles
  tops_[o].tile_off = (u32)ttiles_.size();
  if (check_tensor_vector_size(shape, dt_, mem, vs) != CANON_OK) throw ModelError("an operand is not canonical");
  const u32 from = mem_has_layout(mem) ? tiled_layouts_(sh, lay) : 0;
  u32 c = 0;
  for (int d = 0; d < shape.n; d++)
    for (u32 e = 1; e < shape[d]; e *= 2, c++) {
      Shape tile = shape;
      tile[d] = e;
      u32 entry = mem_has_layout(mem) ? tiled_[from + c] : (DPT_APPLIES | DPT_OK | lay);   // RF: no layout to change
      if ((entry & DPT_OK) && check_tensor_vector_size(tile, dt_, mem, vs) != CANON_OK) entry &= DPT_APPLIES;
      if (entry & DPT_OK) {
        const u32 to = op_id_(tshapes_[sh].child[c], mem, vs, entry & 0x3FFFFFFFu);
        if (to > 0x3FFFFFFFu) throw ModelError("too many operands");
        entry = (entry & (DPT_OK | DPT_APPLIES)) | to;
      } else {
        entry &= DPT_APPLIES;
      }
      ttiles_.push_back(entry);
    }
}

void OpTables::close_operands_() {
  for (u32 o = 0; o < tops_.size(); o++) tabulate_op_(o);
}

u32 OpTables::fam_id_(u8 kind, u8 dtype, const Shape& s) {
  const u64 key = fam_key(kind, dtype, s);
  const size_t at = probe(fam_tab_, fams.size(), mix(2, key), [&](u32 i) { return fam_keys_[i] == key; },
                          [&](u32 i) { return mix(2, fam_keys_[i]); });
  if (fam_tab_[at]) return fam_tab_[at] - 1;
  if (s.n > 8 || ((kind == K_MATMUL || kind == K_MATMUL_ACCUM) && s.n != 4)) throw ModelError("bad Spec shape");
  const u32 id = (u32)fams.size();
  if (id >= DP_NO_FAM) throw ModelError("too many families for the factored planner");
  fam_tab_[at] = id + 1;
  fam_keys_.push_back(key);
  fams.emplace_back();
  DpFam f;
  memset(&f, 0, sizeof(f));
  f.kind = kind;
  f.dtype = dtype;
  f.nd = s.n;
  f.nops = (u8)kind_operand_count((SpecKind)kind);
  LogicalSpec l;
  l.kind = (SpecKind)kind;
  l.spec_shape = s;
  for (int d = 0; d < s.n; d++) f.logs[d] = (u8)log2_of(s[d]);
  f.accum = f.fill = DP_NO_FAM;
  std::vector<u16> child;
  for (int j = 0; j < f.nops; j++) {
    const Shape os = l.operand_shape(j);
    f.shape[j] = (u16)shape_id_(os);
    f.move[j] = (u16)(kind == K_MOVE ? id : fam_id_(K_MOVE, dtype, os));
  }
  if (kind == K_MATMUL) {
    f.accum = (u16)fam_id_(K_MATMUL_ACCUM, dtype, s);
    f.fill = (u16)fam_id_(K_FILL_ZERO, dtype, l.operand_shape(2));
  }
  u32 at_child = 0;
  for (int d = 0; d < s.n; d++) {
    f.child_at[d] = (u8)at_child;
    for (u32 e = 1; e < s[d]; e *= 2, at_child++) {
      Shape t = s;
      t[d] = e;
      child.push_back((u16)fam_id_(kind, dtype, t));
    }
  }
  f.child_off = (u32)fam_child.size();
  fam_child.insert(fam_child.end(), child.begin(), child.end());
  fams[id] = f;
  return id;
}

void OpTables::start_() {
  for (int k = 0; k < NMEM; k++) top_code[k] = limit_code(k, AVX2_MAX_MEM[k]);
}

void OpTables::build_precompute(u32 size, Through through, const std::vector<Dtype>& dtypes) {
  start_();
  if (dtypes.empty()) throw ModelError("no dtypes");
  dt_ = dtypes[0];
  for (Dtype d : dtypes)
    if (dtype_size(d) != dtype_size(dt_)) throw ModelError("dtypes of several sizes");
  // families of the bounds' task points: every shape up to the bound's (space.hpp, goal_phases)
  for (auto& phase : goal_phases(size, through, dtypes))
    for (const Bound& b : phase) {
      Shape s = b.spec_shape;
      std::vector<u32> logs(s.n, 0);
      for (;;) {
        for (int d = 0; d < s.n; d++) s[d] = 1u << logs[d];
        const int kinds = b.kind == K_MATMUL ? 2 : 1;
        for (int k = 0; k < kinds; k++) fam_seed_.push_back(fam_id_(k ? (u8)K_MATMUL_ACCUM : (u8)b.kind, b.dtype, s));
        int d = 0;
        while (d < s.n && (2u << logs[d]) > b.spec_shape[d]) logs[d++] = 0;
        if (d == s.n) break;
        logs[d]++;
      }
    }
  // the variants of an operand in any memory, the same wherever the operand occurs
  goal_lists_.resize(tshapes_.size());
  for (u64 f : fam_seed_)
    for (int j = 0; j < fams[f].nops; j++) {
      const u32 sh = fams[f].shape[j];
      if (!goal_lists_[sh].empty()) continue;
      // (what aux_variants lists per memory: the layouts are the same in every memory that has any)
      const Shape shape = tshapes_[sh].s;
      goal_lists_[sh].push_back(op_id_(sh, RF, 0, layout_id_(Layout())));
      std::vector<u32> vs;
      for (u32 b : mem_vector_bytes(VRF))
        if (check_tensor_vector_size(shape, dt_, VRF, b / dtype_size(dt_)) == CANON_OK) vs.push_back(b / dtype_size(dt_));
      for (const Layout& l : all_layouts_for_shape(shape, dt_))
        for (int contig = 0; contig <= l.n; contig++) {
          Aux a;
          a.mem = GL;
          a.layout = l;
          a.layout.contig = (u8)contig;
          if (!aux_is_canonical(a, shape)) continue;
          const u32 id = layout_id_(a.layout);
          goal_lists_[sh].push_back(op_id_(sh, GL, 0, id));
          goal_lists_[sh].push_back(op_id_(sh, L1, 0, id));
          for (u32 v : vs) goal_lists_[sh].push_back(op_id_(sh, VRF, (u8)v, id));
        }
    }
  close_operands_();
  finish_();
}

void OpTables::build_goals(const std::vector<LogicalSpec>& goals) {
  start_();
  if (goals.empty()) throw ModelError("no goals");
  dt_ = goals[0].dtype;
  std::vector<u64> at;
  at.reserve(goals.size() * 4);
  for (const LogicalSpec& g : goals) {
    if (!g.serial_only) throw ModelError("only serial-only Specs are tabulated");
    if (dtype_size(g.dtype) != dtype_size(dt_)) throw ModelError("dtypes of several sizes");
    const u32 f = fam_id_(g.kind, g.dtype, g.spec_shape);
    at.push_back(f);
    for (int j = 0; j < 3; j++) at.push_back(j < g.nops() ? op_id_(fams[f].shape[j], g.aux[j]) : 0);
  }
  close_operands_();
  finish_();
  for (size_t k = 0; k < at.size(); k += 4) {
    const DpFam& f = fams[at[k]];
    seeds.push_back(dp_pack((u32)at[k], loc_[at[k + 1]], f.nops > 1 ? loc_[at[k + 2]] : 0, f.nops > 2 ? loc_[at[k + 3]] : 0));
  }
}

void OpTables::finish_() {
  // ---- operands of a shape in key order ----
  const u32 n_ops = (u32)tops_.size(), n_shapes = (u32)tshapes_.size();
  if (layouts_.size() > 0xFFFF || n_shapes > 0xFFFF) throw ModelError("too many layouts or shapes for the factored planner");
  loc_.assign(n_ops, 0);
  shapes.resize(n_shapes);
  ops.resize(n_ops);
  auxes.resize(n_ops);
  moves.resize(tmoves_.size());
  tiles.resize(ttiles_.size());
  struct Ordered { u8 bytes[4 + 4 * MAX_PHYS]; u32 len, id; };
  std::vector<Ordered> order;
  size_t tab = 64;
  while (tab < (size_t)n_ops * 2) tab *= 2;
  find_tab_.assign(tab, 0);
  u32 lo = 0;
  for (u32 s = 0; s < n_shapes; s++) {
    const std::vector<u32>& members = tshapes_[s].ops;
    if (members.size() > 0xFFFF) throw ModelError("too many operands of one shape for the factored planner");
    order.resize(members.size());
    for (size_t k = 0; k < members.size(); k++) {
      order[k].id = members[k];
      order[k].len = (u32)aux_bytes(tops_[members[k]].aux, order[k].bytes);
    }
    std::sort(order.begin(), order.end(), [](const Ordered& a, const Ordered& b) {
      const int c = memcmp(a.bytes, b.bytes, std::min(a.len, b.len));
      return c != 0 ? c < 0 : a.len < b.len;
    });
    DpShape& d = shapes[s];
    memset(&d, 0, sizeof(d));
    d.op_lo = lo;
    d.cnt = (u32)members.size();
    d.rank = tshapes_[s].s.n;
    u32 at = 0;
    for (int k = 0; k < d.rank; k++) {
      d.logs[k] = (u8)log2_of(tshapes_[s].s[k]);
      d.sum += d.logs[k];
      d.tile_at[k] = (u8)at;
      at += d.logs[k];
    }
    for (size_t k = 0; k < order.size(); k++) {
      const TmpOp& t = tops_[order[k].id];
      loc_[order[k].id] = (u32)k;
      for (int m = t.aux.mem + 1; m < 5; m++) d.start[m] = (u16)(k + 1);
      auxes[lo + k] = t.aux;
      size_t i = bytes_hash(s, order[k].bytes, order[k].len) & (tab - 1);
      while (find_tab_[i]) i = (i + 1) & (tab - 1);
      find_tab_[i] = lo + (u32)k + 1;
    }
    lo += d.cnt;
  }
  for (u32 i = 0; i < n_ops; i++) {
    const TmpOp& t = tops_[i];
    DpOp& d = ops[shapes[t.shape].op_lo + loc_[i]];
    d.moves_off = t.moves_off;
    d.tile_off = t.tile_off;
    if (t.n_actions > 0xFFFF) throw ModelError("too many Moves of one operand");
    d.n_moves = (u16)t.n_moves;
    d.n_actions = (u16)t.n_actions;
    d.layout_id = (u16)t.layout_id;
    d.rm_loc = (u16)loc_[t.rm];
    d.cost = t.cost;
    d.mem = (u8)t.aux.mem;
    d.vs = t.aux.vector_size;
    d.flags = t.flags;
    d.pad = 0;
  }
  for (size_t i = 0; i < tmoves_.size(); i++) {
    const TmpMove& t = tmoves_[i];
    moves[i] = DpMove{t.imm, t.units, t.rel, (u16)loc_[t.to], t.mem, t.thr, t.miss, 0};
  }
  for (size_t i = 0; i < ttiles_.size(); i++)
    tiles[i] = (ttiles_[i] & DPT_OK) ? ((ttiles_[i] & (DPT_OK | DPT_APPLIES)) | loc_[ttiles_[i] & 0x3FFFFFFFu]) : (ttiles_[i] & DPT_APPLIES);

  // ---- positions: (family, level rank) slices in id order ----
  struct Slice { u64 order; std::string bytes; u32 fam, level, size; };
  std::vector<Slice> sl;
  u32 max_nm = 0;
  for (const DpOp& o : ops) max_nm = std::max<u32>(max_nm, o.n_moves);
  for (u32 fi = 0; fi < fams.size(); fi++) {
    DpFam& f = fams[fi];
    u32 sum = 0, max_log = 0;
    std::string bytes;
    bytes.push_back((char)f.dtype);
    bytes.push_back((char)f.nd);
    for (int d = 0; d < f.nd; d++) {
      sum += f.logs[d];
      max_log = std::max<u32>(max_log, f.logs[d]);
      bytes.push_back((char)((1u << f.logs[d]) & 0xff));
      bytes.push_back((char)((1u << f.logs[d]) >> 8));
    }
    max_records = std::max(max_records, f.nops * max_nm + (max_log + 1) * std::max<u32>(f.nd, 3) + 4u + max_log);
    const DpShape& s0 = shapes[f.shape[0]];
    u32 c0[4], c1[4] = {0, 0, 0, 0}, c2[4] = {0, 0, 0, 0};
    for (int m = 0; m < 4; m++) {
      c0[m] = s0.start[m + 1] - s0.start[m];
      if (f.nops > 1) c1[m] = shapes[f.shape[1]].start[m + 1] - shapes[f.shape[1]].start[m];
      if (f.nops > 2) c2[m] = shapes[f.shape[2]].start[m + 1] - shapes[f.shape[2]].start[m];
    }
    if (f.nops == 3)
      for (int x = 0; x < 7; x++) {
        u64 r = 0;
        for (int m1 = 0; m1 < 4; m1++) {
          f.Q[x][m1] = (u32)r;
          if (x - m1 >= 0 && x - m1 < 4) r += (u64)c1[m1] * c2[x - m1];
        }
        if (r > 0xFFFFFFFFull) throw ModelError("too many positions for the factored planner");
        f.R[x] = (u32)r;
      }
    const int levels = f.nops == 3 ? 10 : 4;
    for (int L = 0; L < levels; L++) {
      u64 size = 0;
      if (f.nops == 1) size = c0[L];
      else if (f.nops == 2) size = (u64)s0.start[L] * c1[L] + (u64)c0[L] * s0.start[L + 1];
      else
        for (int m0 = 0; m0 < 4; m0++) {
          f.base[L][m0] = (u32)size;   // the slice's own base is added below
          if (L - m0 >= 0 && L - m0 < 7) size += (u64)c0[m0] * f.R[L - m0];
        }
      if (size > 0xFFFFFFF0ull) throw ModelError("too many positions for the factored planner");
      if (size == 0) continue;
      sl.push_back(Slice{(u64)f.kind << 32 | (u64)sum << 8 | (u64)L, bytes, fi, (u32)L, (u32)size});
    }
  }
  std::sort(sl.begin(), sl.end(), [](const Slice& a, const Slice& b) { return a.order != b.order ? a.order < b.order : a.bytes < b.bytes; });
  u64 pos = 0;
  for (size_t k = 0; k < sl.size(); k++) {
    if (k == 0 || sl[k].order != sl[k - 1].order) {
      stage_base.push_back((u32)pos);
      stage_key.push_back((u32)(sl[k].order >> 32) << 16 | (u32)(sl[k].order & 0xFFFF));
    }
    DpFam& f = fams[sl[k].fam];
    for (int m0 = 0; m0 < 4; m0++) f.base[sl[k].level][m0] = (f.nops == 3 ? f.base[sl[k].level][m0] : 0) + (u32)pos;
    pos += sl[k].size;
    if (pos > 0xFFFFFF00ull) throw ModelError("too many positions for the factored planner");
  }
  if (pos > (1u << 29)) throw ModelError("too many positions for the factored planner");   // 8 bytes of queue each
  n_positions = (u32)pos;

  // ---- precompute goals: products of the operands' variants ----
  if (!fam_seed_.empty()) {
    std::vector<u32> list_at(n_shapes, 0);
    for (u32 s = 0; s < goal_lists_.size(); s++) {
      list_at[s] = (u32)lists.size();
      for (u32 o : goal_lists_[s]) lists.push_back((u16)loc_[o]);
    }
    const u32 chunk = 4096;
    for (u64 f : fam_seed_) {
      DpProduct p;
      memset(&p, 0, sizeof(p));
      p.fam = (u32)f;
      u64 total = 1;
      for (int j = 0; j < 3; j++) {
        p.n[j] = 1;
        if (j >= fams[f].nops) continue;
        p.list[j] = list_at[fams[f].shape[j]];
        p.n[j] = (u32)goal_lists_[fams[f].shape[j]].size();
        total *= p.n[j];
      }
      for (u64 at = 0; at < total; at += chunk) {
        p.first = (u32)at;
        p.count = (u32)std::min<u64>(chunk, total - at);
        products.push_back(p);
      }
    }
  }
}

// ---- lookups ---------------------------------------------------------------------------------

u32 OpTables::find_op_(u32 shape, u64 h, const u8* bytes, u32 len) const {
  const size_t mask = find_tab_.size() - 1;
  for (size_t i = h & mask; find_tab_[i]; i = (i + 1) & mask) {
    const u32 o = find_tab_[i] - 1;
    if (o < shapes[shape].op_lo || o >= shapes[shape].op_lo + shapes[shape].cnt) continue;
    u8 own[4 + 4 * MAX_PHYS];
    if ((u32)aux_bytes(auxes[o], own) == len && memcmp(own, bytes, len) == 0) return o - shapes[shape].op_lo;
  }
  return 0xFFFFFFFFu;
}

bool OpTables::locate_blob(const u8* s, size_t len, u64* out) const {
  if (len < 4 || s[0] > K_MATMUL || s[2] != 1 || s[3] > MAX_RANK || fam_tab_.empty()) return false;
  const u32 nd = s[3];
  if (len < 4 + 2 * nd) return false;
  u64 key = nd | (u64)s[0] << 40 | (u64)s[1] << 44;
  for (u32 d = 0; d < nd; d++) {
    const u32 v = s[4 + 2 * d] | (u32)s[5 + 2 * d] << 8;
    if (v == 0 || (v & (v - 1)) || v > (1u << 15)) return false;
    key |= (u64)log2_of(v) << (4 + 4 * d);
  }
  const size_t mask = fam_tab_.size() - 1;
  size_t i = mix(2, key) & mask;
  while (fam_tab_[i] && fam_keys_[fam_tab_[i] - 1] != key) i = (i + 1) & mask;
  if (!fam_tab_[i]) return false;
  const u32 fi = fam_tab_[i] - 1;
  const DpFam& f = fams[fi];
  size_t p = 4 + 2 * nd;
  u32 loc[3] = {0, 0, 0};
  for (int j = 0; j < f.nops; j++) {
    if (p + 4 > len || s[p + 2] > MAX_PHYS) return false;
    const u32 n = 4 + 4 * (u32)s[p + 2];
    if (p + n > len) return false;
    loc[j] = find_op_(f.shape[j], bytes_hash(f.shape[j], s + p, n), s + p, n);
    if (loc[j] == 0xFFFFFFFFu) return false;
    p += n;
  }
  if (p != len) return false;
  if (f.kind == K_MOVE) {   // equal contiguous layouts are stored row-major
    const DpOp &a = ops[shapes[f.shape[0]].op_lo + loc[0]], &b = ops[shapes[f.shape[1]].op_lo + loc[1]];
    if (a.layout_id == b.layout_id && (a.flags & DPO_CONTIG)) { loc[0] = a.rm_loc; loc[1] = b.rm_loc; }
  }
  *out = dp_pack(fi, loc[0], loc[1], loc[2]);
  return true;
}

bool OpTables::locate(const LogicalSpec& ls, u64* out) const {
  char kb[LogicalSpec::MAX_KEY];
  const int kl = ls.key_into(kb);
  return locate_blob(reinterpret_cast<const u8*>(kb), (size_t)kl, out);
}

LogicalSpec OpTables::spec_of(u64 packed) const {
  const DpFam& f = fams[packed >> 48];
  LogicalSpec l;
  l.kind = (SpecKind)f.kind;
  l.dtype = (Dtype)f.dtype;
  l.serial_only = true;
  l.spec_shape.n = f.nd;
  for (int d = 0; d < f.nd; d++) l.spec_shape[d] = 1u << f.logs[d];
  for (int j = 0; j < f.nops; j++) l.aux[j] = auxes[shapes[f.shape[j]].op_lo + ((packed >> (32 - 16 * j)) & 0xFFFF)];
  return l;
}

}  // namespace mrl
