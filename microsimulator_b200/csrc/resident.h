// The contact solve with its whole system resident in shared memory.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "batch.h"
#include "solve.h"

namespace msb {

// What a resident solve needs beside the descriptor's system.
struct ResidentArrays {
  const std::uint32_t* places;  // per side (row << 1 | side): its entry's place in the incidence
  std::uint32_t* slot_of;       // per entry: CTA << 16 | slot in that CTA's shared memory
  unsigned long long* inbox;    // grid form: (round, side term) words, `stride` per CTA
  ulonglong2* records;          // grid form: two sets of a record of sums per CTA
  std::uint32_t stride;
  const std::uint32_t* crowded;  // not zero: a body has too many entries (null: not known)
  // Bodies in the order in which CTAs take them, and the entries before each
  // in that order (bodies + 1); null: by slot.
  const std::uint32_t* order;
  const std::uint32_t* order_offsets;
};

constexpr std::uint32_t kResidentMaxCtas = 160;  // grid form at most
constexpr std::uint32_t kResidentWords = 4;                        // 16-byte words a record

// What the device takes: the largest cluster, and the CTAs of a cooperative
// grid (0: none).
struct ResidentLimits {
  int cluster = 0;
  int grid = 0;
};
ResidentLimits resident_limits();

// How a system is spread: CTAs in one cluster (grid == false) or over the
// device (grid == true), and lanes per body; ctas == 0: it does not fit.
struct ResidentPlan {
  int ctas = 0;
  bool grid = false;
  int lanes = 1;
};
// By the shared memory the system takes.  Measured on B200, us per iteration
// against the two-pass solve graph's:
//   1,148 rows, 300 bodies      one CTA 3.6, a cluster of 16 3.8; graph 15.6
//   7,000 rows, 1,000 bodies    clusters of 4, 8 and 16 6.6, 5.4 and 4.6, 32
//                               CTAs of a grid 9.3; graph 23.2
//   82,000 rows, 20,011 bodies  148 CTAs 7.6 with 4 lanes a body; graph 18.8
//   247,000 rows, 60,000 bodies 148 CTAs 9.9 with 1 lane a body; graph 23.1
//   221,000 rows, 100,000 bodies in a trap  148 CTAs 8.8; graph 21.7
// (bodies by slot, not in spatial order: 8.4, 15.7 and 15.5; 4 lanes a body
// where 1 is taken: 17.2 and 10.5 in spatial order.)
ResidentPlan resident_plan(const ResidentLimits& limits, std::uint64_t rows, std::uint64_t bodies);
// The bodies along a Morton curve over their centres (16 bits of key; with
// `colony`, colony by colony, at most 65,536), so that a CTA of the grid form
// holds neighbours and few side terms leave it.  `temp` holds
// sort_temp_words(n) words.
void launch_spatial_order(std::uint32_t n, const float4* pos_len, const GridParams* grid, const std::uint32_t* colony,
                          std::uint32_t colonies, std::uint32_t* keys, std::uint32_t* order, std::uint32_t* temp,
                          cudaStream_t stream);
// The entries before each body in `order`; counts: n + 1 words, temp:
// scan_temp_words(n + 1).
void launch_order_offsets(std::uint32_t n, const std::uint32_t* order, const std::uint32_t* offsets,
                          std::uint32_t* counts, std::uint32_t* order_offsets, std::uint32_t* temp,
                          cudaStream_t stream);
// Inbox words per CTA of the grid form.
std::uint32_t resident_stride();
// Runs the whole solve in one launch: bound, initial gaps, every iteration,
// the final multipliers, gaps and response.  desc must hold the reset
// descriptor; `problem` is its host copy.  A system whose shares turn out
// not to fit (a body of more than kResidentDegree entries, an uneven
// split) leaves everything as it was and sets desc->misfit.  Returns a CUDA
// error code.
int launch_resident(const SolveDesc& problem, SolveDesc* desc, const ResidentArrays& arrays, ResidentPlan plan,
                    cudaStream_t stream);
// A batch of independent colonies in one launch: each colony is the job of a
// gang of neighbouring CTAs that holds it, and each CTA takes its jobs in the
// order of `jobs`.  On one cluster of 16 CTAs the largest colony sets a
// solve's time while the other clusters idle (20,000 cells: about 55 us an
// iteration); a gang of 46 CTAs takes 8 us.  64 colonies of 500-20,000 cells:
// solve phase 52 -> 26 ms a step.
struct ResidentJob {
  std::uint32_t colony;
  std::uint32_t first;  // the gang's CTAs: first, first + 1, ...
  std::uint32_t size;
};
struct ResidentBatch {
  const ResidentJob* jobs;
  ResidentGang* gangs;                // one per job, zero at launch
  const std::uint32_t* list_offsets;  // CTAs + 1: each CTA's jobs in `lists`
  const std::uint32_t* lists;
  const std::uint32_t* cell_offsets;
  const std::uint32_t* row_counts;
  const float* tolerance;
  ColonyState* state;  // status kResidentMisfit: the colony's share did not fit, nothing was done
  std::uint32_t* check;
  std::uint32_t* late;  // set once a wait has run out
};
constexpr std::uint32_t kResidentMisfit = 0xFFFFFFFFu;
// CTAs that hold a system.
std::uint32_t resident_ctas(std::uint64_t rows, std::uint64_t bodies);
int launch_resident_batch(const SolveDesc& problem, const ResidentArrays& arrays, const ResidentBatch& batch, int ctas,
                          cudaStream_t stream);

}  // namespace msb
