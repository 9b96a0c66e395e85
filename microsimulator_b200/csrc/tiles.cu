// The Barzilai-Borwein iteration of large systems by tiles of neighbouring
// bodies.
//
// In the two passes of solve.cu each entry of a body gathers its row's
// (multiplier, gap) and scatters its side term, and in a colony whose slots
// follow no spatial order each of those is an L2 sector of its own: about
// 120 G sectors/s, which bounds the body pass (16.6 M a pass of 4.15 M rows:
// 145 us) well below the memory's bandwidth.  Here the system is renumbered
// once per solve: 256 bodies that lie together make a tile, which owns the
// rows of its first bodies, consecutively.  One block takes a tile: it
// projects its rows' multipliers into shared memory, its bodies sum their
// entries from there, put their side terms there, and the block updates its
// rows.  Only rows between tiles (a fifth or so) leave the block: the tile of
// the second body has them as guests, both side terms go to memory, and a
// second, small pass updates them.  Entries lie in groups of eight bodies
// with the tile's bodies by falling entry count, so that the lanes of a warp
// have equal work and no bank conflicts; the copy engine brings a tile's
// entries into shared memory, the next tile's while the rows are updated.
// (Entries loaded into registers by each thread, 8 or 4 at a time, were
// bound by latency: 250 and 197 us a pass at 4.15 M rows.)
//
// At 4.15 M rows over 1 M bodies the tile pass takes 82 us and the boundary
// pass 16 (163 and 31 in the two passes by slot); 153 of the 155 MB it moves
// at 1.66 M rows are what it cannot do without.  Two blocks an SM, the chain
// of each tile's copy, sums, side terms and rows bounds it, not DRAM.  Two
// lanes a body (512 threads) measured 118 us where one measured 111: more
// instructions, no more overlap.  Tiles of 256, 240, 224, 208 and 192 bodies,
// both passes: 91, 93, 79, 81 and 82 us at 1 M random capsules (a third block
// an SM fits from 224 on), 105, 119, 122, 126 and 132 at 1.7 M grown ones, 110,
// 109, 112, 115 and 119 at 1 M settled, 31 to 35 at 300,000: no smaller size
// is better for all of them.
//
// The arithmetic is the two passes', term by term; a body's entries are in
// row order.  Only the FP64 sums are taken in another fixed order.
#include "tiles.h"

#include <algorithm>
#include <cstdint>

#include "device.cuh"
#include "kernels.h"
#include "solve.h"
#include "solve_decide.cuh"
#include "solve_math.cuh"

namespace msb {
namespace {

constexpr int kThreads = kSolveThreads;
static_assert(kThreads == int(kTileBodies), "one thread per body of a tile");
constexpr int kRowBatch = 4;  // rows of a thread whose loads are in flight together
constexpr int kGuests = 2;    // guests of a thread fetched ahead

extern __shared__ __align__(128) unsigned char tile_memory[];

__device__ __forceinline__ void bulk_copy(std::uint32_t to, const void* from, std::uint32_t bytes, std::uint32_t barrier) {
  if (bytes == 0u) return;
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(to), "l"(from),
      "r"(bytes), "r"(barrier)
      : "memory");
}

// What a tile consists of, and this thread's body in it.
struct Tile {
  std::uint32_t r0, rows, g0, guests, at, slots;
  std::uint32_t degree, slot;
  __device__ __forceinline__ void load(const TileArrays& t, std::uint32_t tile, std::uint32_t bodies) {
    r0 = t.row_base[tile];
    rows = t.row_base[tile + 1] - r0;
    g0 = t.guest_base[tile];
    guests = t.guest_base[tile + 1] - g0;
    at = t.slot_base[tile];
    slots = t.slot_base[tile + 1] - at;
    const std::uint32_t place = tile * kTileBodies + threadIdx.x;
    degree = place < bodies ? t.degree[place] : 0u;
    slot = (place < bodies ? t.group[place / 8] : 0u) + threadIdx.x % 8;
  }
  // The rows' range widened to 16-byte boundaries: where the first row lies
  // in it, and its bytes.
  __device__ __forceinline__ std::uint32_t skip() const { return r0 & 1u; }
  __device__ __forceinline__ std::uint32_t row_bytes() const { return ((skip() + rows + 1u) & ~1u) * 8u; }
};

// A tile's copies by the copy engine (thread 0) complete one phase of
// `barrier`: its entries, then its rows' iterate and constants.
__device__ __forceinline__ void fetch_entries(const Tile& tile, const float4* a, const float4* b, std::uint32_t to_a,
                                              std::uint32_t to_b, std::uint32_t barrier) {
  const std::uint32_t bytes = 16 * tile.slots;
  asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(barrier), "r"(2 * bytes) : "memory");
  bulk_copy(to_a, a + tile.at, bytes, barrier);
  bulk_copy(to_b, b + tile.at, bytes, barrier);
}
__device__ __forceinline__ void fetch_rows(const Tile& tile, const float2* iterate, const float2* constants,
                                           std::uint32_t to_iterate, std::uint32_t to_constants, std::uint32_t barrier) {
  const std::uint32_t bytes = tile.row_bytes();
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(barrier), "r"(2 * bytes) : "memory");
  bulk_copy(to_iterate, iterate + (tile.r0 - tile.skip()), bytes, barrier);
  bulk_copy(to_constants, constants + (tile.r0 - tile.skip()), bytes, barrier);
}
__device__ __forceinline__ bool entries_there(std::uint32_t barrier, std::uint32_t phase, std::uint32_t limit) {
  for (std::uint32_t polls = 0; polls < limit; ++polls) {
    std::uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(barrier), "r"(phase)
        : "memory");
    if (done != 0u) return true;
  }
  return false;
}

template <int Tag, int PerSm>
__global__ void __launch_bounds__(kThreads, PerSm) tile_pass_kernel(SolveDesc* desc, int fixed_mode,
                                                                    std::uint32_t wait_polls) {
  const SolveDesc& d = *desc;
  const std::uint32_t mode = fixed_mode >= 0 ? std::uint32_t(fixed_mode) : d.mode;
  if (fixed_mode < 0 && mode == 1 && d.proceed == 0u) return;  // an unrolled pair after convergence
  // A local copy: the descriptor may change under the stores below, for all
  // the compiler knows.
  const TileArrays t = d.tiles;
  // Of the tiled system: filling the descriptor for another forgets the tiles.
  // (Two blocks an SM leave no register over: this count among TileArrays, or
  // the polls in a variable, took a pass of 4.15 M rows from 84 to 96 us.)
  const std::uint32_t bodies = d.body_count;
  const bool project = mode == 1;
  const float alpha = d.step;
  const float dt = d.dt;
  std::uint32_t* check = &desc->check_status;
  float4* const a = reinterpret_cast<float4*>(tile_memory + 128);
  float4* const b = a + t.max_slots;
  const std::uint32_t row_words = (t.max_rows + 3u) & ~1u;
  float2* const iterate = reinterpret_cast<float2*>(b + t.max_slots);
  float2* const constants = iterate + row_words;
  float2* const side = constants + row_words;
  float* const multiplier = reinterpret_cast<float*>(side + t.max_locals);
  const auto shared_at = [](const void* p) { return static_cast<std::uint32_t>(__cvta_generic_to_shared(p)); };
  const std::uint32_t barrier = shared_at(tile_memory);
  // Each load is issued a phase or a tile before its value is needed: what
  // the tile after the next consists of, the next tile's guests, then their
  // iterates.  (With the next tile's alone looked up, its guests' chain of
  // three loads was 4,500 of a tile's 9,600 cycles.)
  Tile now{}, next{}, after{};
  std::uint32_t guest_row[kGuests] = {}, next_row[kGuests] = {};
  float2 guest[kGuests] = {};
  const auto guest_rows = [&](const Tile& tile, std::uint32_t (&row)[kGuests]) {
#pragma unroll
    for (int i = 0; i < kGuests; ++i) {
      const std::uint32_t g = threadIdx.x + i * kThreads;
      if (g < tile.guests) row[i] = t.guests[tile.g0 + g];
    }
  };
  const auto guest_values = [&](const Tile& tile, const std::uint32_t (&row)[kGuests]) {
#pragma unroll
    for (int i = 0; i < kGuests; ++i) {
      if (threadIdx.x + i * kThreads < tile.guests) guest[i] = t.iterate[row[i]];
    }
  };
  std::uint32_t tile = blockIdx.x;
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(barrier), "r"(1u) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (tile < t.tiles) {
    now.load(t, tile, bodies);
    if (threadIdx.x == 0) {
      fetch_entries(now, t.a, t.b, shared_at(a), shared_at(b), barrier);
      fetch_rows(now, t.iterate, t.constants, shared_at(iterate), shared_at(constants), barrier);
    }
    guest_rows(now, guest_row);
    guest_values(now, guest_row);
    if (tile + gridDim.x < t.tiles) next.load(t, tile + gridDim.x, bodies);
  }
  std::uint32_t phase = 0;
  PassSums sums;
  for (; tile < t.tiles; tile += gridDim.x) {
    const bool more = tile + gridDim.x < t.tiles;
    if (more) guest_rows(next, next_row);
    if (tile + 2 * gridDim.x < t.tiles) after.load(t, tile + 2 * gridDim.x, bodies);
    const std::uint32_t skip = now.skip();
    const std::uint32_t place = tile * kTileBodies + threadIdx.x;
    const bool live = place < bodies;
    float4 body_a, body_b;
    if (live) {
      body_a = __ldcs(&t.body_a[place]);
      body_b = __ldcs(&t.body_b[place]);
    }
    const auto projected = [&](float2 q) { return project ? smax(0.0f, q.x - alpha * q.y) : q.x; };
#pragma unroll
    for (int i = 0; i < kGuests; ++i) {
      const std::uint32_t g = threadIdx.x + i * kThreads;
      if (g < now.guests) multiplier[now.rows + g] = projected(guest[i]);
    }
    for (std::uint32_t g = threadIdx.x + kGuests * kThreads; g < now.guests; g += kThreads) {
      multiplier[now.rows + g] = projected(t.iterate[t.guests[now.g0 + g]]);
    }
    const bool there = entries_there(barrier, phase, wait_polls);
    // The multipliers of the tile's rows, projected; a constraint row's
    // second side adds nothing.
    for (std::uint32_t j = threadIdx.x; j < now.rows; j += kThreads) {
      multiplier[j] = projected(iterate[skip + j]);
      side[j].y = -0.0f;
    }
    if (__syncthreads_or(!there) != 0) {
      if (threadIdx.x == 0) {
        raise_status(check, kStatusIterations);
        // Sums that are not finite end the solve (decide): a further iteration
        // could wait as long again.
        for (int k = 0; k < 5; ++k) d.partials[5 * blockIdx.x + k] = 0.0;
        // The block keeps its shared memory until the copies into it are done.
        entries_there(barrier, phase, kWaitPolls);
      }
      return;
    }
    phase ^= 1u;
    if (live) {
      const std::uint32_t locals = now.rows + now.guests;
      float w[6] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
      float load = 0.0f;
#pragma unroll 4
      for (std::uint32_t k = 0; k < now.degree; ++k) {
        const float4 ea = a[now.slot + 8 * k], eb = b[now.slot + 8 * k];
        const std::uint32_t row = __float_as_uint(eb.w) >> 1;
        const float m = index_ok(row, locals, check) ? multiplier[row] : 0.0f;
        // A zero multiplier adds +-0 to sums that start at +0, which leaves
        // their bits as skipping it would.
        w[0] += m * ea.x;
        w[1] += m * ea.y;
        w[2] += m * ea.z;
        w[3] += m * ea.w;
        w[4] += m * eb.x;
        w[5] += m * eb.y;
        load += eb.z * m;
      }
      float v[6];
      float rate;
      respond(d, d.has_drift ? t.order[place] : 0u, body_a, body_b, w, load, v, rate);
#pragma unroll 4
      for (std::uint32_t k = 0; k < now.degree; ++k) {
        const float4 ea = a[now.slot + 8 * k], eb = b[now.slot + 8 * k];
        const std::uint32_t at = __float_as_uint(eb.w);
        if (index_ok(at >> 1, locals, check)) reinterpret_cast<float*>(side)[at] = side_term(ea, eb, v, rate);
      }
    }
    __syncthreads();
    // The next tile's entries and guests come while this one's rows are
    // updated.
#pragma unroll
    for (int i = 0; i < kGuests; ++i) {
      const std::uint32_t g = threadIdx.x + i * kThreads;
      if (g < now.guests) t.second[guest_row[i]] = side[now.rows + g].y;
    }
    for (std::uint32_t g = threadIdx.x + kGuests * kThreads; g < now.guests; g += kThreads) {
      t.second[t.guests[now.g0 + g]] = side[now.rows + g].y;
    }
    if (more) {
      if (threadIdx.x == 0) fetch_entries(next, t.a, t.b, shared_at(a), shared_at(b), barrier);
      guest_values(next, next_row);
    }
#pragma unroll 2
    for (std::uint32_t j = threadIdx.x; j < now.rows; j += kThreads) {
      const float2 q = iterate[skip + j], c = constants[skip + j], s = side[j];
      if (__float_as_int(c.y) < 0) {
        t.first[now.r0 + j] = s.x;
      } else {
        const float m = multiplier[j];
        const float gn = c.x + dt * (s.x + s.y) + c.y * m;
        sums.add(project, q, m, gn);
        t.iterate[now.r0 + j] = make_float2(m, gn);
      }
    }
    __syncthreads();
    if (more && threadIdx.x == 0) {
      fetch_rows(next, t.iterate, t.constants, shared_at(iterate), shared_at(constants), barrier);
    }
    now = next;
    next = after;
#pragma unroll
    for (int i = 0; i < kGuests; ++i) guest_row[i] = next_row[i];
  }
  sums.reduce_to(d.partials + 5 * blockIdx.x);
}

// The rows between tiles; the last block to finish adds every block's sums
// of both passes in block order and decides.
template <int Tag>
__global__ void __launch_bounds__(kThreads) boundary_pass_kernel(SolveDesc* desc, int fixed_mode, int set_condition,
                                                                 int tile_blocks) {
  SolveDesc& d = *desc;
  const std::uint32_t mode = fixed_mode >= 0 ? std::uint32_t(fixed_mode) : d.mode;
  if (fixed_mode < 0 && mode == 1 && d.proceed == 0u) return;
  const TileArrays& t = d.tiles;
  const bool project = mode == 1;
  const float alpha = d.step;
  PassSums sums;
  const std::uint32_t count = t.boundary_count, stride = gridDim.x * blockDim.x;
  const std::uint32_t* __restrict__ list = t.boundary;
  const float2* __restrict__ constants = t.constants;
  const float* __restrict__ first = t.first;
  const float* __restrict__ second = t.second;
  float2* iterate = t.iterate;
  for (std::uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x; i0 < count; i0 += kRowBatch * stride) {
    std::uint32_t r[kRowBatch];
    float2 q[kRowBatch], c[kRowBatch];
    float term[kRowBatch];
#pragma unroll
    for (int k = 0; k < kRowBatch; ++k) r[k] = list[smin(i0 + k * stride, count - 1)];
#pragma unroll
    for (int k = 0; k < kRowBatch; ++k) {
      q[k] = iterate[r[k]];
      c[k] = constants[r[k]];
      term[k] = first[r[k]] + second[r[k]];
    }
#pragma unroll
    for (int k = 0; k < kRowBatch; ++k) {
      if (i0 + k * stride < count) {
        const float m = project ? smax(0.0f, q[k].x - alpha * q[k].y) : q[k].x;
        const float gn = c[k].x + d.dt * term[k] + fabsf(c[k].y) * m;
        sums.add(project, q[k], m, gn);
        iterate[r[k]] = make_float2(m, gn);
      }
    }
  }
  sums.reduce_to(d.partials + 5 * (tile_blocks + blockIdx.x));
  __threadfence();
  __shared__ bool last;
  if (threadIdx.x == 0) last = atomicAdd(&d.ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  const std::uint32_t proceed = decide(d, mode, tile_blocks + gridDim.x);
  if (threadIdx.x == 0 && set_condition) cudaGraphSetConditional(cudaGraphConditionalHandle(d.handle), proceed);
}

__global__ void unpack_tiles_kernel(const SolveDesc* desc) {
  const SolveDesc& d = *desc;
  const TileArrays& t = d.tiles;
  for (std::uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < d.row_count; r += gridDim.x * blockDim.x) {
    const float2 q = t.iterate[r];
    const std::uint32_t i = t.row_of[r];
    d.multipliers[i] = q.x;
    d.gaps[i] = q.y;
    d.iterate[i] = q;
  }
}

// ------------------------------------------------------------- preparation

// One block per tile: its bodies by falling entry count (ties in spatial
// order), their groups' slots and the tile's.
__global__ void __launch_bounds__(kThreads) tile_order_kernel(std::uint32_t n, const std::uint32_t* __restrict__ spatial,
                                                              const std::uint32_t* __restrict__ offsets,
                                                              const std::uint32_t* __restrict__ keyed_offsets,
                                                              BodyArrays bodies, TileBuild out) {
  __shared__ std::uint32_t degrees[kTileBodies];
  __shared__ std::uint32_t sorted[kTileBodies];
  const std::uint32_t first = blockIdx.x * kTileBodies;
  const std::uint32_t count = smin(kTileBodies, n - first);
  std::uint32_t b = 0, degree = 0;
  if (threadIdx.x < count) {
    b = spatial[first + threadIdx.x];
    degree = offsets[b + 1] - offsets[b];
    if (degree > kTileDegree) out.report[0] = 1u;
    degree = smin(degree, kTileDegree);
  }
  degrees[threadIdx.x] = degree;
  sorted[threadIdx.x] = 0u;
  __syncthreads();
  if (threadIdx.x < count) {
    std::uint32_t rank = 0;
    for (std::uint32_t j = 0; j < count; ++j) {
      const std::uint32_t other = degrees[j];
      rank += other > degree || (other == degree && j < threadIdx.x) ? 1u : 0u;
    }
    const std::uint32_t place = first + rank;
    sorted[rank] = degree;
    out.order[place] = b;
    out.place_of[b] = place;
    out.degree[place] = std::uint8_t(degree);
    out.body_a[place] = bodies.a[b];
    out.body_b[place] = bodies.b[b];
    out.row_counts[place] = keyed_offsets[b + 1] - keyed_offsets[b];
  }
  __syncthreads();
  if (threadIdx.x < kTileBodies / 8) {
    const std::uint32_t slots = 8 * sorted[8 * threadIdx.x];
    std::uint32_t x = slots;
    for (int o = 1; o < 32; o <<= 1) {
      const std::uint32_t u = __shfl_up_sync(0xFFFFFFFFu, x, o);
      if (int(threadIdx.x) >= o) x += u;
    }
    if (8 * threadIdx.x < count) out.group[first / 8 + threadIdx.x] = x - slots;
    if (threadIdx.x == kTileBodies / 8 - 1) {
      out.tile_slots[blockIdx.x] = x;
      atomicMax(&out.report[1], x);
    }
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
    out.tile_slots[gridDim.x] = 0u;
    out.row_counts[n] = 0u;
  }
}

// One block per tile: its rows in the tiles' numbering, those within the tile
// before its boundary rows (whose arrays the boundary pass then reads in whole
// stretches), with their constants and iterate.
__global__ void __launch_bounds__(kThreads) tile_rows_kernel(std::uint32_t n, std::uint32_t rows,
                                                             const uint2* __restrict__ slots,
                                                             const float2* __restrict__ constants,
                                                             const std::uint32_t* __restrict__ keyed_offsets,
                                                             const std::uint32_t* __restrict__ keyed_rows,
                                                             const float* __restrict__ multipliers,
                                                             const float2* __restrict__ iterate, TileBuild out) {
  __shared__ std::uint32_t warp_sums[2][kThreads / 32];
  const std::uint32_t tile = blockIdx.x, place = tile * kTileBodies + threadIdx.x;
  const std::uint32_t r0 = out.row_start[tile * kTileBodies];
  const std::uint32_t count = place < n ? out.row_counts[place] : 0u;
  const std::uint32_t from = place < n ? keyed_offsets[out.order[place]] : 0u;
  const auto crosses = [&](std::uint32_t row) {
    const std::uint32_t second = slots[row].y;
    return second != kInvalidSlot && out.place_of[second] / kTileBodies != tile;
  };
  std::uint32_t crossing = 0;
  for (std::uint32_t k = 0; k < count; ++k) crossing += crosses(keyed_rows[from + k]) ? 1u : 0u;
  // Exclusive sums over the block of the rows within and across.
  const std::uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  std::uint32_t sum[2] = {count - crossing, crossing};
  for (int o = 1; o < 32; o <<= 1) {
    for (auto& x : sum) {
      const std::uint32_t u = __shfl_up_sync(0xFFFFFFFFu, x, o);
      if (int(lane) >= o) x += u;
    }
  }
  if (lane == 31u) {
    warp_sums[0][warp] = sum[0];
    warp_sums[1][warp] = sum[1];
  }
  __syncthreads();
  std::uint32_t within = r0 + sum[0] - (count - crossing), across = r0 + sum[1] - crossing;
  for (std::uint32_t w = 0; w < kThreads / 32; ++w) {
    if (w < warp) {
      within += warp_sums[0][w];
      across += warp_sums[1][w];
    }
    across += warp_sums[0][w];
  }
  for (std::uint32_t k = 0; k < count; ++k) {
    const std::uint32_t row = keyed_rows[from + k];
    const bool boundary = crosses(row);
    const std::uint32_t at = boundary ? across++ : within++;
    const float2 c = constants[row];
    out.row_of[at] = row;
    out.new_of[row] = at;
    out.constants[at] = make_float2(c.x, boundary ? -c.y : c.y);
    out.iterate[at] = multipliers != nullptr ? make_float2(multipliers[row], 0.0f) : iterate[row];
    out.flags[at] = boundary ? 1u : 0u;
  }
  if (threadIdx.x == 0) {
    out.row_base[tile] = r0;
    if (tile == gridDim.x - 1) {
      out.row_base[tile + 1] = out.row_start[n];
      out.flags[rows] = 0u;
    }
  }
}

// Each place's entries of rows that other tiles own.
__global__ void tile_guests_kernel(std::uint32_t n, IncidenceArrays incidence, TileBuild out) {
  for (std::uint32_t place = blockIdx.x * blockDim.x + threadIdx.x; place <= n; place += gridDim.x * blockDim.x) {
    std::uint32_t count = 0;
    if (place < n) {
      const std::uint32_t tile = place / kTileBodies;
      const std::uint32_t r0 = out.row_base[tile], r1 = out.row_base[tile + 1];
      const std::uint32_t begin = incidence.offsets[out.order[place]];
      const std::uint32_t degree = out.degree[place];
      for (std::uint32_t k = 0; k < degree; ++k) {
        const std::uint32_t row = out.new_of[__float_as_uint(incidence.b[begin + k].w) >> 1];
        count += row < r0 || row >= r1 ? 1u : 0u;
      }
    }
    out.guest_counts[place] = count;
  }
}

__global__ void tile_entries_kernel(std::uint32_t n, IncidenceArrays incidence, TileBuild out) {
  for (std::uint32_t place = blockIdx.x * blockDim.x + threadIdx.x; place <= n; place += gridDim.x * blockDim.x) {
    const std::uint32_t tile = place / kTileBodies;
    if (place == n) {
      out.guest_base[(n + kTileBodies - 1) / kTileBodies] = out.guest_start[n];
      continue;
    }
    const std::uint32_t r0 = out.row_base[tile], r1 = out.row_base[tile + 1];
    const std::uint32_t g0 = out.guest_start[tile * kTileBodies];
    if (place % kTileBodies == 0) {
      out.guest_base[tile] = g0;
      atomicMax(&out.report[2], r1 - r0);
      atomicMax(&out.report[3], r1 - r0 + out.guest_start[smin(n, place + kTileBodies)] - g0);
    }
    const std::uint32_t slot = out.slot_base[tile] + out.group[place / 8] + place % 8;
    const std::uint32_t begin = incidence.offsets[out.order[place]];
    const std::uint32_t degree = out.degree[place];
    std::uint32_t guest = out.guest_start[place];
    for (std::uint32_t k = 0; k < degree; ++k) {
      const float4 b = incidence.b[begin + k];
      const std::uint32_t side = __float_as_uint(b.w);
      const std::uint32_t row = out.new_of[side >> 1];
      std::uint32_t local = row - r0;
      if (row < r0 || row >= r1) {
        out.guests[guest] = row;
        local = r1 - r0 + guest - g0;
        ++guest;
      }
      out.a[slot + 8 * k] = incidence.a[begin + k];
      out.b[slot + 8 * k] = make_float4(b.x, b.y, b.z, __uint_as_float(local << 1 | (side & 1u)));
    }
  }
}

__global__ void boundary_list_kernel(std::uint32_t rows, const std::uint32_t* __restrict__ flags,
                                     const std::uint32_t* __restrict__ positions, std::uint32_t* __restrict__ boundary) {
  for (std::uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x) {
    if (flags[r] != 0u) boundary[positions[r]] = r;
  }
}

int sm_count() {
  int device = 0, sms = kSmCount;
  if (cudaGetDevice(&device) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  return sms;
}

}  // namespace

void launch_tile_build(std::uint32_t n, std::uint32_t rows, const std::uint32_t* spatial_order, const uint2* slots,
                       const IncidenceArrays& incidence, const BodyArrays& bodies, const std::uint32_t* keyed_offsets,
                       const std::uint32_t* keyed_rows, const float* multipliers, const float2* iterate,
                       const TileBuild& out, std::uint32_t* temp, cudaStream_t stream) {
  const std::uint32_t tiles = (n + kTileBodies - 1) / kTileBodies;
  cudaMemsetAsync(out.report, 0, 4 * sizeof(std::uint32_t), stream);
  tile_order_kernel<<<tiles, kThreads, 0, stream>>>(n, spatial_order, incidence.offsets, keyed_offsets, bodies, out);
  count_launch();
  exclusive_scan(out.tile_slots, out.slot_base, tiles + 1, temp, stream);
  exclusive_scan(out.row_counts, out.row_start, n + 1ull, temp, stream);
  tile_rows_kernel<<<tiles, kThreads, 0, stream>>>(n, rows, slots, incidence.constants, keyed_offsets, keyed_rows,
                                                   multipliers, iterate, out);
  count_launch();
  tile_guests_kernel<<<grid_for(n + 1ull, 256), 256, 0, stream>>>(n, incidence, out);
  count_launch();
  exclusive_scan(out.guest_counts, out.guest_start, n + 1ull, temp, stream);
  tile_entries_kernel<<<grid_for(n + 1ull, 256), 256, 0, stream>>>(n, incidence, out);
  count_launch();
  exclusive_scan(out.flags, out.positions, rows + 1ull, temp, stream);
  boundary_list_kernel<<<grid_for(rows, 256), 256, 0, stream>>>(rows, out.flags, out.positions, out.boundary);
  count_launch();
}

std::uint64_t tile_shared_bytes(std::uint64_t slots, std::uint64_t rows, std::uint64_t locals) {
  return 128 + 32 * slots + 16 * (rows + 4) + 12 * locals + 16;
}

// 228 KB of shared memory an SM, 1 KB of it the system's for each block; the
// pass's static share is under 1 KB.
std::uint32_t tile_pass_bytes(int per_sm) { return std::uint32_t((std::min(228 / per_sm, 227) - 2) * 1024); }

int tile_blocks_per_sm(std::uint64_t slots, std::uint64_t rows, std::uint64_t locals) {
  for (const int per_sm : {4, 3, 2, 1}) {
    if (tile_shared_bytes(slots, rows, locals) <= tile_pass_bytes(per_sm)) return per_sm;
  }
  return 0;
}

template <int Tag>
static void (*tile_pass(int per_sm))(SolveDesc*, int, std::uint32_t) {
  const auto kernel = per_sm >= 4   ? tile_pass_kernel<Tag, 4>
                      : per_sm == 3 ? tile_pass_kernel<Tag, 3>
                      : per_sm == 2 ? tile_pass_kernel<Tag, 2>
                                    : tile_pass_kernel<Tag, 1>;
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(tile_pass_bytes(per_sm)));
  return kernel;
}

void* tile_pass_function(int per_sm) { return reinterpret_cast<void*>(tile_pass<0>(per_sm)); }
void* boundary_pass_function() { return reinterpret_cast<void*>(boundary_pass_kernel<0>); }
int tile_pass_blocks(int per_sm) { return std::min(sm_count() * per_sm, kMaxPassBlocks / 2); }
int boundary_pass_blocks() {
  int active = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&active, boundary_pass_kernel<0>, kThreads, 0);
  return std::min(sm_count() * std::max(1, active), kMaxPassBlocks / 2);
}

void launch_tile_iteration(SolveDesc* desc, int per_sm, std::uint32_t wait_polls, cudaEvent_t between,
                           cudaStream_t stream) {
  const int blocks = tile_pass_blocks(per_sm);
  const std::uint32_t bytes = tile_pass_bytes(per_sm);
  tile_pass<1>(per_sm)<<<blocks, kThreads, bytes, stream>>>(desc, 1, wait_polls);
  if (between != nullptr) cudaEventRecord(between, stream);
  boundary_pass_kernel<1><<<boundary_pass_blocks(), kThreads, 0, stream>>>(desc, 1, 0, blocks);
  count_launch(2);
}

void launch_unpack_tiles(SolveDesc* desc, int blocks, cudaStream_t stream) {
  unpack_tiles_kernel<<<blocks, kThreads, 0, stream>>>(desc);
  count_launch();
}

}  // namespace msb
