// Planning on the device: launches of the plan kernel (devplan.cu).
#pragma once
#include "devplan.cuh"

namespace mrl {

struct PlanCtl {              // what the plan kernel reports
  u32 queued[4];              // Specs queued by a closure round, by round modulo 4
  u32 rounds;
  u32 n_goals;                // distinct goal Specs
  u32 n_specs;
  unsigned long long n_cands;
};

struct PlanArgs {
  DpTables t;
  const u32* stage_base;
  u32 n_stages;               // possible stages: stage_lo gets n_stages + 1 entries
  const DpProduct* products;
  u32 n_products;
  const u16* lists;
  const u64* seeds;
  u32 n_seeds;
  u32 n_words;
  u32* found;                 // bit per position: the Spec exists; zeroed before the launch, as is:
  PlanCtl* ctl;
  u64* queue;                 // Specs in the order they were found: n_positions entries
  uint2* rank;                // (t.rank, while it is being written)
  u32* stage_lo;              // first id of every possible stage
  unsigned long long* block_sums;
  SpecHdr* hdrs;
  u64* desc;                  // by id: packed family and operand indices
  CandRec* cands;
  u32 cap_specs;
  unsigned long long cap_cands;
  int phases;                 // DPP_*
};
// Parts of the plan kernel. A phase whose output would not fit its buffers (cap_*) is left out, as
// are those behind it; the caller sees the sizes in PlanCtl.
enum { DPP_CLOSURE = 1, DPP_SPECS = 2, DPP_RECORDS = 4 };
constexpr u32 DP_MAX_RECORDS = 512;   // candidates of one Spec the record phase can order

// Co-resident blocks of the plan kernel on the current device, per SM (0: error).
int plan_kernel_blocks_per_sm();
cudaError_t launch_plan_kernel(const PlanArgs& a, int blocks, cudaStream_t stream);
constexpr int kPlanBlock = 128;

}  // namespace mrl
