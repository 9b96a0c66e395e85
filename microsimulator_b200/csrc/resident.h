// The contact solve with its whole system resident in shared memory.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "solve.h"

namespace msb {

// What a resident solve needs beside the descriptor's system.
struct ResidentArrays {
  const std::uint32_t* places;  // per side (row << 1 | side): its entry's place in the incidence
  std::uint32_t* slot_of;       // per entry: CTA << 16 | slot in that CTA's shared memory
  unsigned long long* inbox;    // grid form: (round, side term) words, `stride` per CTA
  ulonglong2* records;          // grid form: two sets of kResidentRecords records of sums
  std::uint32_t stride;
  // Bodies in the order in which CTAs take them, and the entries before each
  // in that order (bodies + 1); null: by slot.
  const std::uint32_t* order;
  const std::uint32_t* order_offsets;
};

constexpr std::uint32_t kResidentMaxCtas = 160;  // grid form at most
constexpr std::uint32_t kResidentRecords = kResidentMaxCtas + 16;  // one per CTA and one per group of CTAs
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
//   82,000 rows, 20,011 bodies  148 CTAs 8.4 with 4 lanes a body, 11.5 with 1
//                               (7.3 in spatial order); graph 18.8
//   247,000 rows, 60,000 bodies 148 CTAs 15.7 with 1 lane a body, 17.2 with 4
//                               (12.6 in spatial order); graph 23.1
//   221,000 rows, 100,000 bodies in a trap  148 CTAs 15.5, 9.0 in spatial
//                               order; graph 21.7
ResidentPlan resident_plan(const ResidentLimits& limits, std::uint64_t rows, std::uint64_t bodies);
// The bodies along a Morton curve over their centres (16 bits of key), so
// that a CTA of the grid form holds neighbours and few side terms leave it.
// `temp` holds sort_temp_words(n) words.
void launch_spatial_order(std::uint32_t n, const float4* pos_len, const GridParams* grid, std::uint32_t* keys,
                          std::uint32_t* order, std::uint32_t* temp, cudaStream_t stream);
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
constexpr std::uint32_t kResidentDegree = 62;

}  // namespace msb
