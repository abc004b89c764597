// Device side of the fill: owns the device copies of a Plan and the row table, and runs the
// stages. Callers hand in host data only.
#pragma once
#include "plan.hpp"
#include "optable.hpp"
#include <cuda_runtime.h>
#include <atomic>
#include <memory>
#include <mutex>
#include <thread>

namespace mrl {

// A node of an implementation tree as the device walks it.
struct WalkNode {
  uint64_t spec;          // packed family and operands (plans made on the device)
  uint32_t id, cpack;     // Spec and limits
  uint32_t main, peaks, tail;
  uint32_t first_child;
  uint16_t n_child, status;
  uint32_t pad;
};
enum { WALK_OK = 0, WALK_NO_SPEC = 1, WALK_UNSAT = 2, WALK_BAD = 3 };

struct FillStats {
  uint64_t n_rows = 0;          // final table rows
  uint64_t cells_solved = 0;    // working-grid cells solved, all passes
  uint64_t cands_evaluated = 0; // candidate records evaluated
  uint64_t lookups = 0;         // child rows gathered
  // Algorithmic bytes of the finished table: per final row 12 bytes out, 16 per candidate record
  // of its Spec and 16 (index + row) per child of every candidate that fits the row's limits.
  // Working cells that do not survive compaction do not count.
  uint64_t alg_bytes = 0;
  uint64_t passes = 0;          // solve passes over all stages
  uint64_t launches = 0;        // kernel launches
  uint64_t early_cells = 0;     // of cells_solved: cells of the grids of the unordered phase
  uint64_t late_cands = 0;      // of cands_evaluated: by the relaxation sweeps
  uint64_t late_items = 0;      // work items the sweeps evaluated
  uint64_t growths = 0;         // times a buffer had to be enlarged (the stage that asked is solved again)
  uint64_t sweeps = 0;          // relaxation sweeps of the candidates with a same-stage child
  uint64_t grid_syncs = 0;      // team-wide barriers inside the stage kernels
  float fill_ms = 0;            // device time of the whole fill (CUDA events on the launch stream)
  float combine_ms = 0;         // device time inside the solve phases (device timer)
  float early_ms = 0;           // of which the unordered phase
  float phase_ms[8] = {};       // device time by part of the stage kernels (MRL_PH_*)
};

class DeviceFill {
 public:
  DeviceFill();
  ~DeviceFill();
  int init(int device);
  int init_events();   // the part of init a caller with its own stream and buffer needs
  // Memory from cudaMalloc (the default), or carved out of one caller-supplied device buffer
  // that is never grown or freed (attach_buffer before upload).
  void attach_buffer(void* base, size_t bytes, cudaStream_t stream, int device);
  // Copies headers and candidate records to the device and sets up the buffers.
  // Gigabytes of candidate records keep going up in the background, in id order, after upload()
  // has returned: the plan must stay as it is until wait_upload() (a fill waits stage by stage
  // for the records it is about to read, so its first stages overlap the copy).
  // skip_cands: the candidate records are not on this host; the caller fills device_cands()
  // itself (e.g. a broadcast from the rank that planned) and then calls cands_arrived().
  int upload(const Plan& plan, bool skip_cands = false);
  // For tests: records go up in the background whatever their size, in pieces of 64 KB, and fills start with
  // room for a few hundred rows.
  void small_start(bool on) { small_start_ = on; }
  // Plans the job on the device (devplan.cu): ids, headers and candidate records are worked out
  // there from the factored tables. On return the plan's sizes are known; prepare_fill() then does
  // for it what upload() does for a host plan. 1: not covered, or the fixed buffer is too small -
  // plan on the host.
  int plan(const OpTables& tab);
  // What it enqueues may still be under way on return: fills on the same stream follow it, and a caller
  // that may put another stream in its place waits with sync().
  int prepare_fill();
  int sync();
  struct StageIds { uint32_t lo, hi; uint64_t cand_end; uint32_t team; };
  const std::vector<StageIds>& stages() const { return stages_; }
  uint64_t n_goals() const { return n_goals_; }
  uint64_t n_cands() const { return n_cand_bytes_ / sizeof(CandRec); }
  // Rows of Specs of a plan made on the device, by packed family and operands (OpTables::locate);
  // a Spec that does not exist gets aux = 1.
  int lookup_packed(const uint64_t* specs, const uint32_t* cpacks, size_t n, MrlRow* out);
  // The implementation tree of a Spec at given limits, nodes in breadth-first order, from the tables
  // and records on the device. root: a Spec id, or packed family and operands. 1: more nodes than the
  // walk holds.
  int walk(uint64_t root, bool packed, uint32_t cpack, std::vector<WalkNode>& out);
  // The finished table as masks (4 words per Spec), first rows and rows.
  int export_table(uint32_t* masks, uint64_t* first_row, MrlRow* rows);
  // Packed family and operands of every Spec of a plan made on the device.
  int read_specs(uint64_t* out);
  int read_hdrs(SpecHdr* out);
  // Blocks until every candidate record is on the device.
  int wait_upload();
  void* device_cands() const { return d_cands_; }
  uint64_t device_cand_bytes() const { return n_cand_bytes_; }
  // After the caller has written device_cands(): checks every record on the device (child ids
  // inside the plan, kinds and levels in range) and lets fills run.
  int cands_arrived();
  // Runs every stage: at most one launch per stage, no host synchronisation before the end.
  int run();
  // The same one stage at a time, for callers that exchange tables between stages (multi-GPU):
  // begin_fill; per stage solve_stage, [exchange stage_masks], place_stage, [exchange rows];
  // end_fill. All work is enqueued on the stream; place_stage synchronises it once.
  int begin_fill();
  int solve_stage(uint32_t stage);
  int stage_masks(uint32_t stage, void** ptr, uint64_t* bytes);
  int place_stage(uint32_t stage, void** rows_ptr, uint64_t* bytes);
  int end_fill();
  // Run on a caller-owned stream (e.g. the one a collective library orders against).
  int set_stream(cudaStream_t s);
  // Point lookups: rows of (Spec id, packed limit codes).
  int lookup(const uint32_t* spec_ids, const uint32_t* cpacks, size_t n, MrlRow* out);
  int verify(uint64_t n_samples, uint64_t seed, uint64_t* checked, uint64_t* mismatches,
             uint64_t* first_bad);
  // Order-independent 64-bit checksum of the logical table: per Spec its id, masks and rows in
  // cell order; where the rows lie in the table does not enter.
  int checksum(uint64_t* out);
  // The whole finished table in two copies: headers (masks, first row) and rows.
  int read_table(SpecHdr* hdrs_out, MrlRow* rows_out);
  // Replaces the table by a saved one (hdrs as read_table gave them).
  int load_table(const SpecHdr* hdrs, const MrlRow* rows, uint64_t n_rows);
  int read_hdr(uint32_t spec, SpecHdr* out);
  int read_rows(uint64_t first, uint64_t n, MrlRow* out);
  void release();
  const char* error() const { return err_; }
  const FillStats& stats() const { return stats_; }
  uint64_t h2d_bytes() const { return h2d_bytes_; }
  MrlRow* device_rows() const { return d_rows_; }
  cudaStream_t stream() const { return stream_; }
  int device() const { return device_; }
  uint32_t n_specs() const { return n_specs_; }

 private:
  // A device buffer that stays from one plan to the next. A context keeps no buffer of more than 256 MB
  // and four times what its present plan asks for, and what it does keep is given back before it reports
  // that the device is out of memory.
  struct DevBuf { void* p = nullptr; size_t cap = 0; };
  int reserve_(DevBuf& b, size_t bytes, bool give_back = true);
  static bool oversized_(const DevBuf& b, size_t bytes);
  void drop_(DevBuf& b);
  int drop_all_();   // buffers and the plan in them
  int alloc_(void** p, size_t bytes);
  void begin_plan_();
  int plan_(const OpTables& tab);
  int upload_(const Plan& plan, bool skip_cands);
  int working_buffers_(bool sharded_mine, uint32_t world);
  int launch_stages_(uint32_t from, uint32_t to, int team, int blocks, bool solve, bool place);
  int blocks_of_(int team) const;
  int launch_solve_(uint32_t stage, bool place_too);
  int launch_place_(uint32_t stage);
  int read_ctl_();                       // device control block -> h_ctl_ (synchronises the stream)
  int grow_after_error_(uint32_t bits);  // enlarges the buffers a failed stage asked for
  int wait_cands_(uint64_t upto_bytes);  // until the candidate bytes [0, upto_bytes) are on the device
  void take_stats_();
  int too_large_();

  int device_ = 0;
  bool fixed_ = false;            // carved from an attached buffer: no growth
  bool small_start_ = false;
  unsigned char* buf_ = nullptr;  // attached buffer
  size_t buf_bytes_ = 0, buf_off_ = 0;
  // buffers, and what lies in them
  DevBuf b_ctl_, b_hdrs_, b_cands_, b_spec_, b_stage_specs_, b_mine_, b_stages_, b_items_, b_temp_, b_rows_, b_lookup_;
  DevBuf b_tables_, b_bits_, b_rank_, b_desc_, b_stage_lo_;   // of planning on the device
  SpecHdr* d_hdrs_ = nullptr;
  CandRec* d_cands_ = nullptr;
  uint4* d_rmask_ = nullptr;
  uint8_t* d_mine_ = nullptr;
  uint32_t* d_minsat_ = nullptr; // by Spec id: lower corner of the satisfiable region
  void* d_sspec_ = nullptr;      // by position in the stage being solved: StageSpec
  uint4* d_changed_[3] = {};     // by position in the stage being solved: what a relaxation sweep changed
  WorkItem* d_items_ = nullptr;  // pieces of grids, handed out to warps by the solve phases
  MrlRow* d_rows_ = nullptr;     // the table
  MrlRow* d_temp_ = nullptr;     // working grids of the stage being solved (temp_cap_ rows), then as many rows for the grids of the unordered phase
  unsigned long long* d_block_sums_ = nullptr;
  FillCtl* d_ctl_ = nullptr;
  std::vector<StageIds> stages_;
  uint32_t top_pack_ = 0;
  uint64_t n_goals_ = 0;
  // the tables of a plan made on the device: what lookups address with
  struct DevTables;
  std::unique_ptr<DevTables> tab_;
  void* h_stage_ = nullptr;      // pinned staging for tables, plan results and lookups
  size_t h_stage_bytes_ = 0;
  int reserve_host_(size_t bytes);
  int read_bulk_(void* out, const void* src, size_t bytes);
  std::vector<unsigned char> h_pageable_;   // h_stage_ of a fixed buffer
  template <class Fill, class Launch>
  int lookup_batches_(size_t n, size_t query_bytes, MrlRow* out, Fill fill, Launch launch);
  FillCtl* h_ctl_ = nullptr;     // pinned, or &ctl_pageable_ when nothing may be allocated
  FillCtl ctl_pageable_;
  uint32_t n_specs_ = 0, max_stage_ = 1;
  uint64_t row_cap_ = 0, temp_cap_ = 0, item_cap_ = 0;
  uint64_t h2d_bytes_ = 0;
  uint64_t n_cand_bytes_ = 0;
  bool cands_present_ = false;   // the device candidate records are complete and checked
  bool filling_ = false;
  int coop_blocks_ = 0;          // co-resident blocks of the stage kernel on this device
  int plan_blocks_ = 0;          // ... of the plan kernel, per SM
  int n_sm_ = 0;
  FillStats stats_;
  cudaStream_t stream_ = nullptr;
  bool own_stream_ = false;
  cudaEvent_t ev0_ = nullptr, ev1_ = nullptr;
  std::mutex lookup_mu_;
  // background candidate upload: pieces handed out in order to a few copying threads
  std::vector<std::thread> up_threads_;
  std::unique_ptr<std::atomic<uint8_t>[]> up_done_;   // by piece
  std::atomic<size_t> up_next_{0};
  std::atomic<int> up_err_{0};                        // cudaError_t of the first failed copy
  size_t up_pieces_ = 0, up_piece_bytes_ = 0, up_ready_ = 0;   // up_ready_: pieces known complete, a prefix
  char err_[256] = {0};
};

// Size of the fixed device array behind the no-allocation entry point (32 MiB per GPU).
#define MRL_STATIC_SCRATCH_BYTES (32u << 20)

// One whole small fill inside the fixed device array: plan arrays, working buffers, row table
// and lookup staging; no device allocation. See combine.cu.
int fill_static(int device, cudaStream_t stream, const Plan& plan, const uint32_t* spec_ids, const uint32_t* cpacks,
                size_t n, MrlRow* out, char* err, size_t err_len);
// The same with the plan made on the device too; 1: plan on the host.
int fill_static(int device, cudaStream_t stream, const OpTables& tab, const uint64_t* specs, const uint32_t* cpacks,
                size_t n, MrlRow* out, char* err, size_t err_len);

}  // namespace mrl
