// What the passes of the solve share: a block's part of the BB products and
// the decision that follows an iteration.
#pragma once

#include <cstdint>

#include "device.cuh"
#include "solve.h"
#include "solve_math.cuh"
#include "../../include/msb200.h"

namespace msb {

// A thread's BB products, largest residual and finiteness over its rows.
struct PassSums {
  double ss = 0.0, sy = 0.0, yy = 0.0;
  float residual = 0.0f;
  bool finite = true;

  // A row that went from `before` (multiplier, gap) to (m, gap); with
  // `project` a projected step, whose products count.
  __device__ __forceinline__ void add(bool project, float2 before, float m, float gap) {
    residual = smax(residual, row_residual(m, gap));
    finite = finite && isfinite(gap);
    if (project) {
      const double moved = double(m) - double(before.x);
      const double change = double(gap) - double(before.y);
      ss += moved * moved;
      sy += moved * change;
      yy += change * change;
    }
  }
  // The block's five values, reduced in a fixed tree (the whole block).
  __device__ __forceinline__ void reduce_to(double* to) const {
    __shared__ double red[5][kSolveThreads / 32];
    double v[5] = {ss, sy, yy, double(residual), finite ? 1.0 : 0.0};
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
  #pragma unroll
    for (int k = 0; k < 5; ++k) {
      for (int o = 16; o > 0; o >>= 1) {
        const double other = __shfl_down_sync(0xFFFFFFFFu, v[k], o);
        v[k] = k < 3 ? v[k] + other : (k == 3 ? fmax(v[k], other) : fmin(v[k], other));
      }
      if (lane == 0) red[k][warp] = v[k];
    }
    __syncthreads();
    if (threadIdx.x < 5) {
      const int k = threadIdx.x;
      double r = red[k][0];
      for (int w = 1; w < kSolveThreads / 32; ++w) {
        r = k < 3 ? r + red[k][w] : (k == 3 ? fmax(r, red[k][w]) : fmin(r, red[k][w]));
      }
      to[k] = r;
    }
    __syncthreads();
  }
};

// One block combines the partials of `blocks` blocks in block order (so the
// result does not depend on scheduling), sets the next step length, the
// status and whether to go on (d.proceed), as one iteration of
// iterate_contact_steps does (cpp/core/contact_solver.hpp:66-82); mode 0
// judges the initial multipliers.  Returns d.proceed (thread 0).
__device__ __forceinline__ std::uint32_t decide(SolveDesc& d, std::uint32_t mode, std::uint32_t blocks) {
  __shared__ double red[5][kSolveThreads / 32];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  double t[5] = {0.0, 0.0, 0.0, 0.0, 1.0};
  for (std::uint32_t p = threadIdx.x; p < blocks; p += blockDim.x) {
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const double x = __ldcg(&d.partials[5 * p + k]);
      t[k] = k < 3 ? t[k] + x : (k == 3 ? fmax(t[k], x) : fmin(t[k], x));
    }
  }
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    for (int o = 16; o > 0; o >>= 1) {
      const double other = __shfl_down_sync(0xFFFFFFFFu, t[k], o);
      t[k] = k < 3 ? t[k] + other : (k == 3 ? fmax(t[k], other) : fmin(t[k], other));
    }
  }
  __syncthreads();
  if (lane == 0) {
#pragma unroll
    for (int k = 0; k < 5; ++k) red[k][warp] = t[k];
  }
  __syncthreads();
  if (threadIdx.x != 0) return 0;
  double total[5];
  for (int k = 0; k < 5; ++k) {
    total[k] = red[k][0];
    for (int w = 1; w < kSolveThreads / 32; ++w) {
      total[k] = k < 3 ? total[k] + red[k][w] : (k == 3 ? fmax(total[k], red[k][w]) : fmin(total[k], red[k][w]));
    }
  }
  d.ticket = 0;
  const float reported = total[4] > 0.5 ? float(total[3]) : __int_as_float(0x7FC00000);
  d.residual = reported;
  std::uint32_t proceed = 0;
  if (mode == 0) {
    const float bound = __uint_as_float(__ldcg(&d.bound_bits));
    d.bound = bound;
    d.iterations = 0;
    if (!isfinite(bound) || !(bound > 0.0f)) {
      d.status = 3;  // no positive diagonal: an invalid system
    } else if (!isfinite(reported)) {
      d.status = MSB_SOLVE_BREAKDOWN;
    } else if (reported <= d.tolerance) {
      d.status = MSB_SOLVE_CONVERGED;
    } else {
      d.status = MSB_SOLVE_ITERATION_LIMIT;
      d.step = 1.0f / bound;
      proceed = d.max_iterations > 0 ? 1u : 0u;
    }
    d.mode = 1;
  } else {
    const std::uint32_t iteration = d.iterations + 1;
    d.iterations = iteration;
    if (!isfinite(reported)) {
      d.status = MSB_SOLVE_BREAKDOWN;
    } else if (!(reported > d.tolerance)) {
      d.status = MSB_SOLVE_CONVERGED;
    } else {
      d.step = next_step(d.step, total[0], total[1], total[2], iteration);
      d.status = MSB_SOLVE_ITERATION_LIMIT;
      proceed = iteration < d.max_iterations ? 1u : 0u;
    }
  }
  d.proceed = proceed;
  return proceed;
}

}  // namespace msb
