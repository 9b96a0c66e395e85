// The large contact solve by tiles of neighbouring bodies.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace msb {

struct SolveDesc;
struct RowArrays;
struct IncidenceArrays;
struct BodyArrays;
struct KeyedLists;

constexpr std::uint32_t kTileBodies = 256;
constexpr std::uint32_t kTileDegree = 62;   // entries a body may have

// A system renumbered for the tiled solve.  Places are bodies along the
// substep's spatial order, kTileBodies a tile, within a tile by falling entry
// count; a tile owns the rows whose first body it holds, numbered tile by
// tile ("tile rows").  Rows of other tiles whose second body a tile holds are
// its guests.
struct TileArrays {
  const std::uint32_t* order;      // body of each place
  const std::uint8_t* degree;      // entries of each place
  const std::uint32_t* slot_base;  // per tile: its first entry slot
  const std::uint32_t* group;      // per 8 places: their first slot in the tile
  // Entry k of place p: slot slot_base + group + p % 8 + 8 k.  a = jacobian
  // 0..3, b = jacobian 4, 5, lever, and (row << 1 | side), the row counted in
  // the tile: its own rows, then its guests.
  const float4* a;
  const float4* b;
  const float4* body_a;            // bodies by place
  const float4* body_b;
  const std::uint32_t* row_base;   // tiles + 1: a tile's first row
  const std::uint32_t* guest_base; // tiles + 1: a tile's first guest
  const std::uint32_t* guests;     // tile rows
  const std::uint32_t* row_of;     // per tile row: its row
  const float2* constants;         // offset, compliance (sign bit: a boundary row, second body in another tile)
  float2* iterate;                 // multiplier, gap
  float* first;                    // boundary rows' side terms
  float* second;
  const std::uint32_t* boundary;   // the boundary rows
  std::uint32_t tiles;
  std::uint32_t boundary_count;
  std::uint32_t max_slots;         // of any tile
  std::uint32_t max_rows;          // rows
  std::uint32_t max_locals;        // and rows with guests
};

// Buffers of the preparation; sizes in elements.
struct TileBuild {
  std::uint32_t* order;        // n
  std::uint32_t* place_of;     // n
  std::uint8_t* degree;        // n
  std::uint32_t* tile_slots;   // tiles + 1
  std::uint32_t* slot_base;    // tiles + 1
  std::uint32_t* group;        // n / 8 + 32
  float4* a;                   // tile_slot_capacity
  float4* b;
  float4* body_a;              // n
  float4* body_b;
  std::uint32_t* row_counts;   // n + 1
  std::uint32_t* row_start;    // n + 1
  std::uint32_t* row_base;     // tiles + 1
  std::uint32_t* guest_counts; // n + 1
  std::uint32_t* guest_start;  // n + 1
  std::uint32_t* guest_base;   // tiles + 1
  std::uint32_t* guests;       // rows
  std::uint32_t* row_of;       // rows
  std::uint32_t* new_of;       // rows
  float2* constants;           // rows
  float2* iterate;             // rows
  std::uint32_t* flags;        // rows + 1
  std::uint32_t* positions;    // rows + 1
  std::uint32_t* boundary;     // rows
  std::uint32_t* report;       // 4: a body has too many entries; most slots, rows, rows and guests of a tile
};

// Entry slots at most of `entries` entries over `tiles` tiles: a tile's
// groups of 8 pad at most 8 times its largest degree.
inline std::uint64_t tile_slot_capacity(std::uint64_t entries, std::uint64_t tiles) {
  return entries + tiles * 8 * (kTileDegree + 1);
}

// Renumbers the system of `rows` rows over `n` bodies taken along
// `spatial_order`, with the rows' multipliers (gaps zero) or, where that is
// null, their iterate; `temp`: scan_temp_words(max(n, rows) + 1).  The boundary
// rows' number is then at positions[rows].
void launch_tile_build(std::uint32_t n, std::uint32_t rows, const std::uint32_t* spatial_order, const uint2* slots,
                       const IncidenceArrays& incidence, const BodyArrays& bodies, const std::uint32_t* keyed_offsets,
                       const std::uint32_t* keyed_rows, const float* multipliers, const float2* iterate,
                       const TileBuild& out,
                       std::uint32_t* temp, cudaStream_t stream);

// Shared memory of a tile of at most `slots` slots, `rows` rows and `locals`
// rows and guests, and how many blocks of the tile pass share an SM by it: 4,
// 3, 2 or 1, 0 when it does not fit.  As many as fit: the tile pass of 1 M
// capsules with 4, 3, 2 and 1 took 41, 44, 45 and 70 us at 0.96 M rows, 58, 59,
// 57 and 85 at 1.58 M, with 3, 2 and 1 68, 64 and 95 at 2.17 M, with 2 and 1 69
// and 103 at 2.65 M; of 600,000 with 4, 3, 2 and 1 32, 35, 33 and 51.
std::uint64_t tile_shared_bytes(std::uint64_t slots, std::uint64_t rows, std::uint64_t locals);
int tile_blocks_per_sm(std::uint64_t slots, std::uint64_t rows, std::uint64_t locals);

// The two passes of an iteration (see tiles.cu) for a graph: kernels taking
// (SolveDesc*, int fixed_mode, uint32_t wait_polls) and (SolveDesc*, int
// fixed_mode, int set_condition, int tile_blocks), their grids, and the first one's dynamic
// shared memory, for `per_sm` blocks an SM.
void* tile_pass_function(int per_sm);
void* boundary_pass_function();
int tile_pass_blocks(int per_sm);
std::uint32_t tile_pass_bytes(int per_sm);
int boundary_pass_blocks();

// One more projected iteration of the last system, solved by tiles, for
// timing (launch_iteration's counterpart).
void launch_tile_iteration(SolveDesc* desc, int per_sm, std::uint32_t wait_polls, cudaEvent_t between,
                           cudaStream_t stream);

// The multipliers and gaps a tiled solve reached, by row.
void launch_unpack_tiles(SolveDesc* desc, int blocks, cudaStream_t stream);

}  // namespace msb
