// The device-resident Barzilai-Borwein projected-gradient contact solve.
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "kernels.h"
#include "tiles.h"

namespace msb {

// Rows as structure of arrays (72 bytes per row):
//   a = first jacobian 0..3          b = first jacobian 4, 5, first lever, offset
//   c = second jacobian 0..3         d = second jacobian 4, 5, second lever, compliance
//   slots = (first slot, second slot or kInvalidSlot)
struct RowArrays {
  float4* a;
  float4* b;
  float4* c;
  float4* d;
  uint2* slots;
};

// Bodies (48 bytes per body):
//   a = axis x, y, z, translational mobility
//   b = transverse mobility, axial mobility, nominal elongation rate, 0
//   drift_a / drift_b = drift velocity and angular velocity (w unused)
struct BodyArrays {
  float4* a;
  float4* b;
  float4* drift_a;
  float4* drift_b;
};

// What a set of multipliers does to each body (32 bytes per body):
//   a = velocity x, y, z, loaded elongation rate
//   b = angular velocity x, y, z, axial load
struct ResponseArrays {
  float4* a;
  float4* b;
};

// Per body, its rows in row order (CSR): entry a = jacobian 0..3,
// entry b = jacobian 4, 5, lever, side (bits: row << 1 | 0 for the row's
// first slot, 1 for its second).
// Per row, for the BB passes (null where no BB pass runs on them):
//   constants = (offset, compliance), written with the incidence;
//   sides     = each side's term of the gap rate, jacobian . velocity -
//               lever * elongation rate, indexed by the entries' side bits
//               and written by the body pass.  A constraint row's second
//               side holds -0.0f, which adds nothing: x + -0.0f == x;
//   places    = by side bits, where in the incidence the side's entry is (a
//               constraint row's second side: undefined).
struct IncidenceArrays {
  std::uint32_t* offsets;
  float4* a;
  float4* b;
  float2* constants;
  float2* sides;
  std::uint32_t* places;
};

// Entries a body may have in a resident solve.
constexpr std::uint32_t kResidentDegree = 62;

// Where the CTAs of a resident solve meet: how many hold their shares and how
// many are done, the round they count from (the largest of their own), and
// whether a share did not fit (nothing was done) or a wait ran out.
struct ResidentGang {
  std::uint32_t arrived;
  std::uint32_t left;
  std::uint32_t base;
  std::uint32_t misfit;
  std::uint32_t late;  // of a single system; a batch's is ResidentBatch::late
};

// The ordinary SolveDesc::wait_polls: some seconds of trips to L2 at half a
// microsecond each.
constexpr std::uint32_t kWaitPolls = 1u << 23;

// Everything one solve reads and writes, in device memory at a fixed address
// so that the captured solve graph can be replayed for any system.
struct SolveDesc {
  RowArrays rows;
  BodyArrays bodies;
  IncidenceArrays incidence;
  ResponseArrays response;
  float* multipliers;
  float* gaps;
  // (multiplier, gap) of every row while a solve runs: the body pass
  // gathers both with one load.  The bound pass fills it from `multipliers`;
  // launch_unpack_iterate writes the solution back.
  float2* iterate;
  double* partials;  // 5 doubles per block of the row pass
  std::uint32_t row_count;
  std::uint32_t body_count;
  float dt;
  std::uint32_t law;
  float sensitivity;
  float free_load;
  float stall_load;
  float tolerance;
  std::uint32_t max_iterations;
  std::uint32_t has_drift;  // 0: every drift is zero and the drift arrays are not read
  TileArrays tiles;         // of a tiled solve
  // solver state
  float step;
  float residual;
  float bound;
  std::uint32_t iterations;
  std::uint32_t status;  // msb_solve_status
  std::uint32_t mode;    // 0: evaluate the initial multipliers; 1: iterate
  std::uint32_t ticket;
  std::uint32_t proceed;
  // Written by SolveGraph::launch: the cudaGraphConditionalHandle of the WHILE
  // node, and whether the graph goes on from this state instead of resetting it.
  unsigned long long handle;
  unsigned long long resume;
  std::uint32_t bound_ticket;
  std::uint32_t bound_bits;
  // grid barrier of the fused solve (relax_kernel)
  std::uint32_t barrier_count;
  std::uint32_t barrier_generation;
  std::uint32_t barrier_abort;  // a barrier wait ran out of time: every block stops
  std::uint32_t check_status;   // the first failed check (0: none): a wait that ran out; checked build: an index
  ResidentGang gang;            // the resident solve's
  std::uint32_t wait_polls;     // a 32nd of the polls after which a resident solve's CTAs are late
};

// Every pass reads the tiles' pointers and the state; 8 bytes more before them
// cost 1 us of a 90 us iteration of 4.15 M rows by tiles.
static_assert(offsetof(SolveDesc, tiles) % 16 == 0);

// Builds the incidence of `rows` over `bodies` bodies.  Scratch: `values` holds
// 2 * rows words, `counts` bodies + 1 words (+ 2 with `mark_crowded`), `temp`
// scan_temp_words(bodies + 1) words.  With `mark_crowded`, counts[bodies + 1]
// says whether a body has more than kResidentDegree entries.
void build_incidence(RowArrays rows, std::uint32_t row_count, std::uint32_t body_count, IncidenceArrays incidence,
                     std::uint32_t* values, std::uint32_t* counts, std::uint32_t* temp, cudaStream_t stream,
                     std::uint32_t* status = nullptr, bool mark_crowded = false);

// Stable lists of each first slot's rows (ForceMemory's KeyedRows).
void build_keyed(const uint2* slots, std::uint32_t row_count, std::uint32_t body_count, std::uint32_t* offsets,
                 std::uint32_t* rows_out, std::uint32_t* counts, std::uint32_t* temp, cudaStream_t stream);

// A solve graph for a fixed grid size: bound -> initial gaps -> WHILE
// (not converged) { body pass; row pass }.
class SolveGraph {
 public:
  SolveGraph() = default;
  SolveGraph(const SolveGraph&) = delete;
  SolveGraph& operator=(const SolveGraph&) = delete;
  ~SolveGraph();
  // `tiles_per_sm` > 0: the passes of tiles.cu, which read desc->tiles, with
  // that many blocks an SM and `wait_polls`.  Returns a CUDA error code.
  int create(SolveDesc* desc, int blocks, cudaStream_t stream, int tiles_per_sm = 0,
             std::uint32_t wait_polls = kWaitPolls);
  // With `resume` the solve in the descriptor goes on.
  int launch(cudaStream_t stream, bool resume = false);
  int blocks() const { return blocks_; }
  // Kernel launches of the WHILE node for a solve of `iterations`
  // iterations (whole evaluations of its unrolled body).
  static int loop_launches(std::uint32_t iterations);

 private:
  cudaGraph_t graph_ = nullptr;
  cudaGraphExec_t exec_ = nullptr;
  int blocks_ = 0;
  SolveDesc* desc_ = nullptr;
  unsigned long long handle_ = 0;
};

// The fused solve: bound, initial gaps and every projected iteration in ONE
// cooperative launch of `blocks` co-resident blocks, with two bounded grid
// barriers per iteration (the last block to reach the second combines the
// BB products and decides).  The whole descriptor, state included, must be
// reset before the launch; `problem` is its host copy, passed by value as a
// kernel parameter.  Returns a CUDA error code.
int launch_relax(const SolveDesc& problem, SolveDesc* desc, int blocks, cudaStream_t stream);
// Blocks of relax_kernel that fit on the device at once.
int relax_resident_blocks();
// How long a barrier wait may take before the solve stops with
// barrier_abort set.
constexpr unsigned long long kBarrierTimeoutNs = 5'000'000'000ull;

// Evaluates the response of desc->multipliers once (no solve), as
// evaluate_contact_response does; also the gaps when `with_gaps`.  A solve
// writes no response itself: this evaluation of its final multipliers
// follows it.
void launch_evaluate(SolveDesc* desc, int blocks, bool with_gaps, cudaStream_t stream);
// The multipliers and gaps a solve reached (desc->iterate) into
// desc->multipliers and desc->gaps.
void launch_unpack_iterate(SolveDesc* desc, int blocks, cudaStream_t stream);

// One more projected iteration of the last solved system (body pass then
// row pass), for timing; `between` is recorded between the two passes.
void launch_iteration(SolveDesc* desc, int blocks, cudaEvent_t between, cudaStream_t stream);

constexpr int kSolveThreads = 256;
// Blocks of a BB pass at most: the per-block partials hold this many.
constexpr int kMaxPassBlocks = 1184;

}  // namespace msb
