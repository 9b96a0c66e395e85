// The Barzilai-Borwein contact solve with the system resident in shared
// memory: one launch runs the bound, the initial gaps and every projected
// iteration, and between iterations nothing but side terms and sums moves.
//
// Each CTA holds a contiguous range of bodies and those bodies' incidence
// entries: the jacobian and lever, the row's offset and compliance, and the
// row's (multiplier, gap).  Both bodies of a row keep its multiplier and gap
// and update them with the same operations, so an iteration is
//   send     per body: project its entries' multipliers, sum their wrenches
//            in entry order (the reference's row order), respond, and send
//            each entry's side term of the gap rate to the row's other entry;
//   receive  per entry: own term + received term -> the new gap; the BB
//            products and the residual (rows counted on their first side).
// The arithmetic is that of the two-pass solve (solve.cu), term by term; only
// the FP64 products are summed in another fixed order.
//
// Three forms by size.  One CTA: block barriers.  One cluster: side terms go
// through distributed shared memory, with two hardware cluster barriers per
// iteration.  The whole grid (a cooperative launch): a term for another CTA
// is one 64-bit word (round, value) in that CTA's global inbox, which its
// owner polls; the sums are words of the same kind that every CTA reads and
// adds in CTA order, so no CTA waits for another's decision and no grid
// barrier is needed.  Every wait for a word is bounded (kWaitPolls: seconds),
// and so is a gang's wait for its CTAs to arrive and to leave, which may have
// to finish other systems first (wait_count: minutes, or until another CTA has
// given up).
#include "resident.h"

#include <cooperative_groups.h>

#include <algorithm>
#include <bit>
#include <type_traits>
#include <cstdint>

#include "device.cuh"
#include "kernels.h"
#include "solve_math.cuh"
#include "../../include/msb200.h"

namespace cg = cooperative_groups;

namespace msb {
namespace {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr std::uint32_t kGroup = 8;    // bodies whose entries are interleaved
constexpr std::uint32_t kClasses = 64;  // degree classes of the stable sort
// Shared bytes of an entry (jacobian and lever 32, constants and iterate 16,
// own and received term 8, list of the remote ones 2) and of a body
// (record 32, index 2, degree 1, share of the group offsets).
constexpr std::uint32_t kEntryBytes = 58;
constexpr std::uint32_t kBodyBytes = 36;
constexpr std::uint32_t kNobody = 0xFFFFFFFFu;  // a constraint row's entry sends nothing
constexpr std::uint32_t kRemote = 0x80000000u;

enum Form { kSingle, kCluster, kGrid };
enum Round { kBound, kInitial, kIterate, kFinal };

struct Sums {
  double v[3];          // ss, sy, yy
  std::uint32_t bits;   // largest residual (or bound) as float bits; a NaN's when a gap is not finite
};

struct Shared {
  std::uint16_t histogram[kWarps][kClasses];
  std::uint32_t class_base[kClasses];
  Sums warp[16];   // each warp's sums
  Sums parts[16];  // the cluster's, written by its CTAs
  std::uint32_t round;
  std::uint32_t misfit;
  std::uint32_t remote_count;
  std::uint32_t slots;
  std::uint32_t inbox_at;     // shared address of this CTA's inbox
  std::uint32_t inboxes[16];  // and of every CTA's of the cluster
};

extern __shared__ __align__(16) unsigned char resident_memory[];

// Where a CTA's arrays lie in its dynamic shared memory.
struct Layout {
  std::uint32_t a_at, b_at, c_at, own_at, inbox_at, remote_at;       // by slot
  std::uint32_t body_a_at, body_b_at, body_at, degree_at, group_at;  // by body, by group
  std::uint32_t bodies;
  std::uint32_t slots;
  std::uint32_t first;  // the CTA's first body

  template <class T>
  __device__ __forceinline__ static T& at(std::uint32_t offset, std::uint32_t i) {
    return reinterpret_cast<T*>(resident_memory + offset)[i];
  }
  __device__ __forceinline__ float4& a(std::uint32_t j) const { return at<float4>(a_at, j); }
  // Jacobian 4, 5, lever, where this entry's term goes.
  __device__ __forceinline__ float4& b(std::uint32_t j) const { return at<float4>(b_at, j); }
  // Offset, compliance (sign bit: the row's first side), multiplier, gap.
  __device__ __forceinline__ float4& c(std::uint32_t j) const { return at<float4>(c_at, j); }
  __device__ __forceinline__ float& own(std::uint32_t j) const { return at<float>(own_at, j); }
  __device__ __forceinline__ float& inbox(std::uint32_t j) const { return at<float>(inbox_at, j); }
  __device__ __forceinline__ std::uint16_t& remote(std::uint32_t x) const { return at<std::uint16_t>(remote_at, x); }
  __device__ __forceinline__ float4& body_a(std::uint32_t q) const { return at<float4>(body_a_at, q); }
  __device__ __forceinline__ float4& body_b(std::uint32_t q) const { return at<float4>(body_b_at, q); }
  __device__ __forceinline__ std::uint16_t& body(std::uint32_t q) const { return at<std::uint16_t>(body_at, q); }
  __device__ __forceinline__ std::uint8_t& degree(std::uint32_t q) const { return at<std::uint8_t>(degree_at, q); }
  // First slot of each kGroup bodies.
  __device__ __forceinline__ std::uint32_t& group(std::uint32_t g) const { return at<std::uint32_t>(group_at, g); }
};

// Body q's slots are base_of(q) + kGroup * k, k below its degree; up to its
// group's depth they are padding: zeros that send nothing.
__device__ __forceinline__ std::uint32_t base_of(const Layout& l, std::uint32_t q) {
  return l.group(q / kGroup) + q % kGroup;
}
__device__ __forceinline__ std::uint32_t depth_of(const Layout& l, std::uint32_t q) {
  return l.degree(q - q % kGroup);
}
__device__ __forceinline__ void pad_slot(const Layout& l, std::uint32_t j) {
  l.a(j) = l.c(j) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  l.b(j) = make_float4(0.0f, 0.0f, 0.0f, __uint_as_float(kNobody));
  l.own(j) = l.inbox(j) = 0.0f;
}

__device__ __forceinline__ void put_word(unsigned long long* p, std::uint32_t tag, std::uint32_t value) {
  const unsigned long long w = (static_cast<unsigned long long>(tag) << 32) | value;
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
}
__device__ __forceinline__ unsigned long long get_word(const unsigned long long* p) {
  unsigned long long w;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
  return w;
}
// A double and a 32-bit value with their round as one 128-bit word.
__device__ __forceinline__ void put_wide(ulonglong2* p, std::uint32_t tag, std::uint32_t bits, double v) {
  const unsigned long long hi = (static_cast<unsigned long long>(tag) << 32) | bits;
  asm volatile(
      "{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
      "l"(__double_as_longlong(v)), "l"(hi)
      : "memory");
}
__device__ __forceinline__ ulonglong2 get_wide(const ulonglong2* p) {
  ulonglong2 w;
  asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
               : "=l"(w.x), "=l"(w.y)
               : "l"(p)
               : "memory");
  return w;
}
// Waits until *p carries `tag`; false once the wait has run out.  (A limit
// that is no constant costs more than its comparison: a step of 60,000 cells
// took 7.4 ms for 6.7.)
__device__ __forceinline__ bool wait_word(const unsigned long long* p, std::uint32_t tag, unsigned long long& word) {
  for (std::uint32_t polls = 0; std::uint32_t(word >> 32) != tag; ++polls) {
    if (polls == kWaitPolls) return false;
    word = get_word(p);
  }
  return true;
}

// Waits until *p has reached `count`, a gang's CTAs having arrived or left:
// they may first finish other systems, so the limit is 32 * `limit` polls (by
// default 2^28 of half a microsecond: about two minutes).  False once it has
// run out or another CTA has set *late.
__device__ __forceinline__ bool wait_count(const std::uint32_t* p, std::uint32_t count, std::uint32_t limit,
                                           const std::uint32_t* late) {
  const auto read = [](const std::uint32_t* from) { return *static_cast<const volatile std::uint32_t*>(from); };
  for (std::uint64_t polls = 0; read(p) < count; ++polls) {
    if (polls >= 32ull * limit) return false;
    if (polls > 1024u) {
      if (read(late) != 0u) return false;
      __nanosleep(500);
    }
  }
  return true;
}

__device__ __forceinline__ std::uint32_t cluster_address(std::uint32_t local, std::uint32_t rank) {
  std::uint32_t out;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(local), "r"(rank));
  return out;
}
__device__ __forceinline__ void cluster_store(std::uint32_t address, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(address), "f"(v) : "memory");
}

__device__ __forceinline__ std::uint64_t weight(const std::uint32_t* offsets, std::uint32_t b0, std::uint32_t b) {
  return std::uint64_t(kEntryBytes) * (offsets[b] - offsets[b0]) + std::uint64_t(kBodyBytes) * (b - b0);
}
// The first body of [b0, b1] whose weight reaches `target` (block-wide).
__device__ std::uint32_t find_split(const std::uint32_t* offsets, std::uint32_t b0, std::uint32_t b1,
                                    std::uint64_t target) {
  std::uint32_t lo = b0, hi = b1;
  while (lo < hi) {
    const std::uint32_t step = (hi - lo + kThreads - 1) / kThreads;
    const std::uint64_t p = std::uint64_t(lo) + std::uint64_t(threadIdx.x) * step;
    const int below = __syncthreads_count(p < hi && weight(offsets, b0, std::uint32_t(p)) < target);
    if (below == 0) return lo;
    const std::uint32_t last = lo + std::uint32_t(below - 1) * step;
    hi = smin<std::uint64_t>(hi, std::uint64_t(last) + step);
    lo = last + 1;
  }
  return lo;
}

// The body at a place of the order in which CTAs take them.
__device__ __forceinline__ std::uint32_t body_at(const ResidentArrays& r, std::uint32_t place) {
  return r.order != nullptr ? r.order[place] : place;
}

template <int kForm>
struct Comm {
  std::uint32_t rank, size;
  const ResidentArrays* arrays;
  std::uint32_t first = 0;  // grid form: the first of the gang's CTAs
  std::uint32_t round = 0;  // grid form: tags words, never falls within a launch
  ResidentGang* gang = nullptr;
  std::uint32_t* late = nullptr;   // grid form: set once a CTA has given up a wait
  std::uint32_t wait_polls = 0;

  __device__ void sync_all() const {
    if constexpr (kForm == kCluster) {
      cg::this_cluster().sync();
    } else {
      __syncthreads();
    }
  }
  // Sends a side term to the entry that meta names.
  __device__ __forceinline__ void send(const Layout& l, std::uint32_t meta, float value) const {
    if (meta == kNobody) return;
    if constexpr (kForm == kSingle) {
      l.inbox(meta) = value;
    } else if constexpr (kForm == kCluster) {
      cluster_store(meta, value);
    } else {
      if (meta & kRemote) {
        put_word(arrays->inbox + (meta & ~kRemote), round, __float_as_uint(value));
      } else {
        l.inbox(meta) = value;
      }
    }
  }
  // Every term sent in this round is in its inbox on return.
  __device__ bool exchange(const Layout& l, const Shared& s) const {
    if constexpr (kForm != kGrid) {
      sync_all();
      return true;
    } else {
      const unsigned long long* words = arrays->inbox + std::size_t(first + rank) * arrays->stride;
      bool late = false;
      constexpr int kFlight = 4;
      for (std::uint32_t x0 = threadIdx.x; x0 < s.remote_count; x0 += kFlight * kThreads) {
        unsigned long long w[kFlight];
        std::uint32_t slot[kFlight];
#pragma unroll
        for (int t = 0; t < kFlight; ++t) {
          const std::uint32_t x = x0 + t * kThreads;
          if (x < s.remote_count) {
            slot[t] = l.remote(x);
            w[t] = get_word(words + slot[t]);
          }
        }
#pragma unroll
        for (int t = 0; t < kFlight; ++t) {
          if (x0 + t * kThreads < s.remote_count) {
            late = !wait_word(words + slot[t], round, w[t]) || late;
            l.inbox(slot[t]) = __uint_as_float(std::uint32_t(w[t]));
          }
        }
        if (late) break;
      }
      return __syncthreads_or(late) == 0;
    }
  }
};

// Sums over a warp in a fixed tree: ss in lanes 0-7, sy in lanes 8-15, yy in
// lanes 16-23 of the result, and the largest bits in every lane.  Halving the
// values with the lanes takes 6 double shuffles, not the 15 of three trees.
__device__ __forceinline__ double fold_warp(const Sums& x, std::uint32_t& bits) {
  const std::uint32_t lane = threadIdx.x & 31u;
  const bool upper = (lane & 16u) != 0u, odd = (lane & 8u) != 0u;
  double p = (upper ? x.v[2] : x.v[0]) + __shfl_xor_sync(0xFFFFFFFFu, upper ? x.v[0] : x.v[2], 16);
  const double q = __shfl_xor_sync(0xFFFFFFFFu, x.v[1], 16);
  const double r = upper ? 0.0 : x.v[1] + q;
  p = (odd ? r : p) + __shfl_xor_sync(0xFFFFFFFFu, odd ? p : r, 8);
  for (int o = 4; o > 0; o >>= 1) p += __shfl_xor_sync(0xFFFFFFFFu, p, o);
  bits = __reduce_max_sync(0xFFFFFFFFu, x.bits);
  return p;
}
__device__ __forceinline__ void store_sums(Sums& to, double p, std::uint32_t bits) {
  const std::uint32_t lane = threadIdx.x & 31u;
  if (lane == 24u) to.bits = bits;
  if ((lane & 7u) == 0u && lane < 24u) to.v[lane / 8] = p;
}
// The same of 16 records in shared memory, and its totals in every lane.
__device__ __forceinline__ Sums fold_records(const Sums* records) {
  const std::uint32_t lane = threadIdx.x & 31u, k = lane >> 3, i = lane & 7u;
  double p = k < 3u ? records[i].v[k] + records[i + 8].v[k] : 0.0;
  for (int o = 4; o > 0; o >>= 1) p += __shfl_xor_sync(0xFFFFFFFFu, p, o);
  const std::uint32_t bits = __reduce_max_sync(0xFFFFFFFFu, lane < 16u ? records[lane].bits : 0u);
  return {{__shfl_sync(0xFFFFFFFFu, p, 0), __shfl_sync(0xFFFFFFFFu, p, 8), __shfl_sync(0xFFFFFFFFu, p, 16)}, bits};
}

static_assert(kWarps <= 16, "fold_records reads 16 records");
// CTA `rank`'s record, in one of two alternating sets: a CTA writes a set
// again only after every CTA has read the other, and so has read this one.
__device__ __forceinline__ ulonglong2* record_of(const Comm<kGrid>& comm, std::uint32_t rank) {
  return comm.arrays->records + (std::size_t(comm.round & 1u) * kResidentMaxCtas + comm.first + rank) * kResidentWords;
}
__device__ __forceinline__ bool get_record(const Comm<kGrid>& comm, std::uint32_t rank, Sums& x) {
  const ulonglong2* from = record_of(comm, rank);
  ulonglong2 w[3];
  const auto there = [&] {
    bool all = true;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      w[k] = get_wide(from + k);
      all = all && std::uint32_t(w[k].y >> 32) == comm.round;
    }
    return all;
  };
  for (std::uint32_t polls = 0; !there(); ++polls) {
    if (polls == kWaitPolls) return false;
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) x.v[k] = __longlong_as_double(static_cast<long long>(w[k].x));
  x.bits = std::uint32_t(w[0].y);
  return true;
}

// The sums of every CTA, in a fixed order, in every thread.  False (grid
// form) once a wait has run out.
template <int kForm>
__device__ __forceinline__ bool reduce(const Comm<kForm>& comm, Shared& s, Sums& x) {
  const std::uint32_t lane = threadIdx.x & 31u;
  std::uint32_t bits;
  double p = fold_warp(x, bits);
  store_sums(s.warp[threadIdx.x >> 5], p, bits);
  __syncthreads();
  if constexpr (kForm == kSingle) {
    x = fold_records(s.warp);
  } else if constexpr (kForm == kCluster) {
    if (threadIdx.x < 32) {
      x = fold_records(s.warp);
      if (lane < comm.size) *cg::this_cluster().map_shared_rank(&s.parts[comm.rank], lane) = x;
    }
    comm.sync_all();
    x = fold_records(s.parts);
  } else {
    // Every CTA reads every CTA's record, 32 a warp (a second hop, through
    // sums of 12 CTAs each, took an iteration of 60,000 cells from 9.9 to
    // 12.6 us).
    if (threadIdx.x < 32) {
      x = fold_records(s.warp);
      if (lane < 3u) put_wide(record_of(comm, comm.rank) + lane, comm.round, x.bits, lane == 0u ? x.v[0] : lane == 1u ? x.v[1] : x.v[2]);
    }
    bool late = false;
    x = Sums{{0.0, 0.0, 0.0}, 0u};
    if ((threadIdx.x & ~31u) < comm.size) {
      if (threadIdx.x < comm.size) late = !get_record(comm, threadIdx.x, x);
      p = fold_warp(x, bits);
      store_sums(s.parts[threadIdx.x >> 5], p, bits);
    }
    if (__syncthreads_or(late) != 0) return false;
    x = fold_records(s.parts);
  }
  return true;
}

// A body's wrench and load over its entries in entry order, the body's
// response, and its entries' side terms on their way (kFinal: the response
// written instead), by P lanes per body.  A padding entry or a zero
// multiplier adds +-0 to sums that start at +0, which leaves their bits as
// skipping it would.
//
// P = 1: one thread sums all seven components.  P > 1, for CTAs with few
// bodies: each lane sums 8 / P of the components, each still in entry order,
// the lanes exchange them, and the side terms are dealt out entry by entry.
template <int P, int kForm>
__device__ __forceinline__ void send_sides(const SolveDesc& d, const Layout& l, const Comm<kForm>& comm, int round,
                                           float alpha) {
  constexpr std::uint32_t kPass = kThreads / P;  // bodies a pass
  constexpr int kShare = 8 / P;                  // components a lane
  const std::uint32_t lane = threadIdx.x % P;
  const bool project = round == kIterate;
#pragma unroll 1
  for (std::uint32_t q0 = 0; q0 < l.bodies; q0 += kPass) {
    // Lanes past the last body repeat it (P > 1: the warp exchanges sums).
    const std::uint32_t at = q0 + threadIdx.x / P;
    if (P == 1 && at >= l.bodies) break;
    const std::uint32_t q = smin(at, l.bodies - 1);
    const std::uint32_t depth = depth_of(l, q);
    const std::uint32_t base = base_of(l, q);
    const float4 ba = l.body_a(q);
    const float4 bb = l.body_b(q);
    float v[6] = {};
    float rate = 0.0f;
    if (round != kBound) {
      float w[8] = {};
      if constexpr (P == 1) {
#pragma unroll 1
        for (std::uint32_t k = 0; k < depth; ++k) {
          const std::uint32_t j = base + kGroup * k;
          const float4 ea = l.a(j), eb = l.b(j), c = l.c(j);
          const float m = project ? smax(0.0f, c.z - alpha * c.w) : c.z;
          w[0] += m * ea.x;
          w[1] += m * ea.y;
          w[2] += m * ea.z;
          w[3] += m * ea.w;
          w[4] += m * eb.x;
          w[5] += m * eb.y;
          w[6] += eb.z * m;
        }
      } else {
        const std::uint32_t half = lane / (P / 2);              // 0: components 0-3 (a), 1: 4-6 (b)
        const std::uint32_t part = (lane % (P / 2)) * kShare;   // first component within it
        const std::uint32_t from = (half != 0u ? l.b_at : l.a_at) / (4 * kShare) + part / kShare;
        float mine[kShare] = {};
#pragma unroll 2
        for (std::uint32_t k = 0; k < depth; ++k) {
          const std::uint32_t j = base + kGroup * k;
          const float2 c = Layout::at<float2>(l.c_at, 2 * j + 1);
          float jac[kShare];
          if constexpr (P == 4) {
            const float2 t = Layout::at<float2>(0, from + 2 * j);
            jac[0] = t.x;
            jac[1] = t.y;
          } else {
            jac[0] = Layout::at<float>(0, from + 4 * j);
          }
          const float m = project ? smax(0.0f, c.x - alpha * c.y) : c.x;
#pragma unroll
          for (int i = 0; i < kShare; ++i) mine[i] += m * jac[i];
        }
#pragma unroll
        for (int i = 0; i < 7; ++i) w[i] = __shfl_sync(0xFFFFFFFFu, mine[i % kShare], i / kShare, P);
      }
      const std::uint32_t b = body_at(*comm.arrays, l.first + l.body(q));
      const float wrench[6] = {w[0], w[1], w[2], w[3], w[4], w[5]};
      respond(d, b, ba, bb, wrench, w[6], v, rate);
      if (round == kFinal) {
        if (lane == 0 && at < l.bodies) {
          d.response.a[b] = make_float4(v[0], v[1], v[2], rate);
          d.response.b[b] = make_float4(v[3], v[4], v[5], w[6]);
        }
        continue;
      }
    }
    if (at < l.bodies) {
#pragma unroll 1
      for (std::uint32_t k = lane; k < depth; k += P) {
        const std::uint32_t j = base + kGroup * k;
        const float4 ea = l.a(j), eb = l.b(j);
        const float term = round == kBound ? diagonal(ea, eb, ba, bb) : side_term(ea, eb, v, rate);
        l.own(j) = term;
        comm.send(l, __float_as_uint(eb.w), term);
      }
    }
  }
}

// One entry per thread: the row's gap from both terms, and this CTA's share
// of the sums.  Slots that pad a group hold zeros throughout.
__device__ __forceinline__ Sums receive_sides(const SolveDesc& d, const Layout& l, int round, float alpha) {
  Sums s{{0.0, 0.0, 0.0}, 0u};
  float residual = 0.0f;
  bool finite = true;
  const float dt = d.dt;
  const bool project = round == kIterate;
#pragma unroll 1
  for (std::uint32_t j = threadIdx.x; j < l.slots; j += kThreads) {
    const float4 c = l.c(j);
    const float rate = l.own(j) + l.inbox(j);
    const float compliance = fabsf(c.y);
    if (round == kBound) {
      residual = smax(residual, dt * rate + compliance);
    } else {
      const float m = project ? smax(0.0f, c.z - alpha * c.w) : c.z;
      const float gn = c.x + dt * rate + compliance * m;
      residual = smax(residual, row_residual(m, gn));
      finite = finite && isfinite(gn);
      if (project && __float_as_int(c.y) < 0) {
        const double moved = double(m) - double(c.z);
        const double change = double(gn) - double(c.w);
        s.v[0] += moved * moved;
        s.v[1] += moved * change;
        s.v[2] += change * change;
      }
      *reinterpret_cast<float2*>(&l.c(j).z) = make_float2(m, gn);
    }
  }
  s.bits = finite ? __float_as_uint(residual) : 0x7FC00000u;
  return s;
}

// Loads this CTA's share of bodies [b0, b1).  False when some CTA's share does
// not fit `bytes` of shared memory (in every CTA, s.misfit 1) or the other CTAs
// did not arrive in time (s.misfit 2).  (Returning the outcome itself took the
// one-CTA solves of a 300-cell step from 253 to 269 us: other code.)
template <int kForm>
__device__ bool load_share(const SolveDesc& d, const ResidentArrays& r, Comm<kForm>& comm, Shared& s, Layout& l,
                           std::uint32_t bytes, std::uint32_t b0, std::uint32_t b1, std::uint32_t* check) {
  const std::uint32_t* offsets = r.order != nullptr ? r.order_offsets : d.incidence.offsets;
  const std::uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  std::uint32_t first = b0, last = b1;
  if constexpr (kForm != kSingle) {
    const std::uint64_t total = weight(offsets, b0, b1);
    if (comm.rank > 0) first = find_split(offsets, b0, b1, total * comm.rank / comm.size);
    if (comm.rank + 1 < comm.size) last = find_split(offsets, b0, b1, total * (comm.rank + 1) / comm.size);
    __syncthreads();
  }
  const std::uint32_t bodies = last - first;
  l.first = first;
  l.bodies = bodies;
  const std::uint32_t groups = (bodies + kGroup - 1) / kGroup;
  // Carve the parts that depend on the body count.
  std::uint64_t at = 0;
  const auto carve = [&](std::uint64_t size) {
    const std::uint32_t here = std::uint32_t(at);
    at += (size + 15) & ~std::uint64_t(15);
    return here;
  };
  l.body_a_at = carve(16ull * bodies);
  l.body_b_at = carve(16ull * bodies);
  l.group_at = carve(4ull * groups);
  l.body_at = carve(2ull * bodies);
  l.degree_at = carve(bodies);
  for (std::uint32_t i = threadIdx.x; i < 16; i += kThreads) s.warp[i] = s.parts[i] = Sums{{0.0, 0.0, 0.0}, 0u};
  if (threadIdx.x == 0) {
    const bool crowded = r.crowded != nullptr && *r.crowded != 0u;
    s.misfit = crowded || at > bytes || bodies > 0xFFFFu ? 1u : 0u;
    s.remote_count = 0;
    s.slots = 0;
  }
  for (std::uint32_t i = threadIdx.x; i < kWarps * kClasses; i += kThreads) (&s.histogram[0][0])[i] = 0;
  __syncthreads();
  const bool room = s.misfit == 0;
  __syncthreads();
  if (room) {
    // Bodies by falling degree (a stable counting sort, so that the order of
    // the sums does not depend on scheduling): the 32 bodies of a warp then
    // have nearly the same number of entries.
    const std::uint32_t per = ((bodies + kWarps - 1) / kWarps + 31) & ~31u;
    const std::uint32_t from = smin(bodies, warp * per), to = smin(bodies, from + per);
    for (std::uint32_t i = from; i < to; i += 32) {
      const bool live = i + lane < to;
      std::uint32_t cls = kClasses;
      if (live) {
        const std::uint32_t degree = offsets[first + i + lane + 1] - offsets[first + i + lane];
        if (degree > kResidentDegree) s.misfit = 1u;
        cls = kClasses - 1 - smin(degree, kResidentDegree);
      }
      const std::uint32_t peers = __match_any_sync(0xFFFFFFFFu, cls);
      if (live && lane == std::uint32_t(__ffs(peers) - 1)) s.histogram[warp][cls] += std::uint16_t(__popc(peers));
      __syncwarp();
    }
    __syncthreads();
    if (threadIdx.x < kClasses) {
      std::uint32_t sum = 0;
      for (int w = 0; w < kWarps; ++w) {
        const std::uint32_t n = s.histogram[w][threadIdx.x];
        s.histogram[w][threadIdx.x] = std::uint16_t(sum);
        sum += n;
      }
      s.class_base[threadIdx.x] = sum;
    }
    __syncthreads();
    if (warp == 0) {
      std::uint32_t x = s.class_base[lane], y = s.class_base[lane + 32], sx = x, sy = y;
      for (int o = 1; o < 32; o <<= 1) {
        const std::uint32_t u = __shfl_up_sync(0xFFFFFFFFu, sx, o), v = __shfl_up_sync(0xFFFFFFFFu, sy, o);
        if (int(lane) >= o) {
          sx += u;
          sy += v;
        }
      }
      const std::uint32_t half = __shfl_sync(0xFFFFFFFFu, sx, 31);
      s.class_base[lane] = sx - x;
      s.class_base[lane + 32] = half + sy - y;
    }
    __syncthreads();
    for (std::uint32_t i = from; i < to; i += 32) {
      const bool live = i + lane < to;
      std::uint32_t cls = kClasses, degree = 0;
      if (live) {
        degree = smin(offsets[first + i + lane + 1] - offsets[first + i + lane], kResidentDegree);
        cls = kClasses - 1 - degree;
      }
      const std::uint32_t peers = __match_any_sync(0xFFFFFFFFu, cls);
      if (live) {
        const std::uint32_t rank = __popc(peers & ((1u << lane) - 1u));
        const std::uint32_t q = s.class_base[cls] + s.histogram[warp][cls] + rank;
        l.body(q) = std::uint16_t(i + lane);
        l.degree(q) = std::uint8_t(degree);
      }
      __syncwarp();
      if (live && lane == std::uint32_t(__ffs(peers) - 1)) s.histogram[warp][cls] += std::uint16_t(__popc(peers));
      __syncwarp();
    }
    __syncthreads();
    // Slots of each group: kGroup times the degree of the first, the largest.
    if (warp == 0) {
      std::uint32_t sum = 0;
      for (std::uint32_t g0 = 0; g0 < groups; g0 += 32) {
        const std::uint32_t n = g0 + lane < groups ? kGroup * l.degree(kGroup * (g0 + lane)) : 0u;
        std::uint32_t x = n;
        for (int o = 1; o < 32; o <<= 1) {
          const std::uint32_t u = __shfl_up_sync(0xFFFFFFFFu, x, o);
          if (int(lane) >= o) x += u;
        }
        if (g0 + lane < groups) l.group(g0 + lane) = sum + x - n;
        sum += __shfl_sync(0xFFFFFFFFu, x, 31);
      }
      if (lane == 0) s.slots = sum;
    }
    __syncthreads();
    const std::uint32_t slots = s.slots;
    l.slots = slots;
    l.a_at = carve(16ull * slots);
    l.b_at = carve(16ull * slots);
    l.c_at = carve(16ull * slots);
    l.own_at = carve(4ull * slots);
    l.inbox_at = carve(4ull * slots);
    if (threadIdx.x == 0) s.inbox_at = static_cast<std::uint32_t>(__cvta_generic_to_shared(resident_memory)) + l.inbox_at;
    l.remote_at = carve(kForm == kGrid ? 2ull * slots : 0ull);
    if (threadIdx.x == 0 && (at > bytes || slots > 0xFFFFu || (kForm == kGrid && slots > r.stride))) s.misfit = 1u;
    __syncthreads();
    if (s.misfit == 0) {
      for (std::uint32_t q = threadIdx.x; q < bodies; q += kThreads) {
        const std::uint32_t b = body_at(r, first + l.body(q));
        l.body_a(q) = d.bodies.a[b];
        l.body_b(q) = d.bodies.b[b];
        const std::uint32_t degree = l.degree(q), depth = depth_of(l, q);
        const std::uint32_t base = base_of(l, q);
        const std::uint32_t begin = d.incidence.offsets[b];
        for (std::uint32_t k = 0; k < degree; ++k) {
          const std::uint32_t j = base + kGroup * k;
          const float4 eb = d.incidence.b[begin + k];
          const std::uint32_t side = __float_as_uint(eb.w), row = side >> 1;
          const float2 constants = d.incidence.constants[row];
          l.a(j) = d.incidence.a[begin + k];
          l.b(j) = eb;
          const float compliance = fabsf(constants.y);  // -0 included
          l.c(j) = make_float4(constants.x, (side & 1u) ? compliance : -compliance, d.multipliers[row], 0.0f);
          l.own(j) = 0.0f;
          l.inbox(j) = 0.0f;
          r.slot_of[begin + k] = comm.rank << 16 | j;
        }
        for (std::uint32_t k = degree; k < depth; ++k) {
          pad_slot(l, base + kGroup * k);
        }
      }
      // The last group's missing bodies.
      if (bodies % kGroup != 0) {
        const std::uint32_t there = bodies % kGroup, missing = kGroup - there, depth = depth_of(l, bodies - there);
        for (std::uint32_t i = threadIdx.x; i < missing * depth; i += kThreads) {
          pad_slot(l, l.group(groups - 1) + kGroup * (i / missing) + there + i % missing);
        }
      }
    }
  }
  // Every CTA's slots are known (or one does not fit) from here on.
  if constexpr (kForm == kGrid) {
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
      ResidentGang& gang = *comm.gang;
      if (s.misfit != 0) atomicExch(&gang.misfit, 1u);
      atomicMax(&gang.base, comm.round);
      __threadfence();
      atomicAdd(&gang.arrived, 1u);
      const bool late = !wait_count(&gang.arrived, comm.size, comm.wait_polls, comm.late);
      __threadfence();
      if (*static_cast<volatile std::uint32_t*>(&gang.misfit) != 0u) s.misfit = 1u;
      if (late) s.misfit = 2u;
      s.round = *static_cast<volatile std::uint32_t*>(&gang.base);
    }
    __syncthreads();
    comm.round = s.round;
  } else if constexpr (kForm == kCluster) {
    __threadfence();
    comm.sync_all();
    const bool misfit = __syncthreads_or(threadIdx.x < comm.size &&
                                         *cg::this_cluster().map_shared_rank(&s.misfit, threadIdx.x) != 0u) != 0;
    if (threadIdx.x < comm.size) s.inboxes[threadIdx.x] = *cg::this_cluster().map_shared_rank(&s.inbox_at, threadIdx.x);
    comm.sync_all();
    if (misfit) s.misfit = 1u;
    __syncthreads();
  } else {
    __syncthreads();
  }
  if (s.misfit != 0) return false;
  // Where each entry's side terms go: the other entry of its row.
  for (std::uint32_t q = threadIdx.x; q < bodies; q += kThreads) {
    const std::uint32_t degree = l.degree(q);
    const std::uint32_t base = base_of(l, q);
    for (std::uint32_t k = 0; k < degree; ++k) {
      const std::uint32_t j = base + kGroup * k;
      const std::uint32_t side = __float_as_uint(l.b(j).w);
      std::uint32_t meta = kNobody;
      if (!index_ok(side >> 1, d.row_count, check)) {
        l.inbox(j) = -0.0f;
      } else if ((side & 1u) != 0u || d.rows.slots[side >> 1].y != kInvalidSlot) {
        const std::uint32_t place = r.places[side ^ 1u];
        const std::uint32_t to =
            index_ok(place, 2ull * d.row_count, check) ? __ldcg(&r.slot_of[place]) : comm.rank << 16 | j;
        const std::uint32_t cta = to >> 16, slot = to & 0xFFFFu;
        if constexpr (kForm == kSingle) {
          meta = slot;
        } else if constexpr (kForm == kCluster) {
          meta = cluster_address(s.inboxes[cta] + 4 * slot, cta);
        } else if (cta == comm.rank) {
          meta = slot;
        } else {
          meta = kRemote | ((comm.first + cta) * r.stride + slot);
          l.remote(atomicAdd(&s.remote_count, 1u)) = std::uint16_t(j);
        }
      } else {
        // A constraint row has no second side: -0.0f adds nothing.
        l.inbox(j) = -0.0f;
      }
      l.b(j).w = __uint_as_float(meta);
    }
  }
  __syncthreads();
  return true;
}

struct Report {
  float step, residual, bound;
  std::uint32_t iterations, status;
};
enum Outcome { kSolved, kMisfit, kLate };

// The whole solve of bodies [b0, b1) by the CTAs of `comm`.
template <int kForm, int P>
__device__ __forceinline__ Outcome resident_solve(const SolveDesc& d, const ResidentArrays& r, Comm<kForm>& comm,
                                                  Shared& s, std::uint32_t bytes, std::uint32_t b0, std::uint32_t b1,
                                                  float tolerance, std::uint32_t* check, Report& report) {
  Layout l{};
  if (!load_share(d, r, comm, s, l, bytes, b0, b1, check)) return kForm == kGrid && s.misfit == 2u ? kLate : kMisfit;
  // Every thread takes the same decisions from the same sums.  The rounds
  // share one copy of the code: what a round executes is fetched once per
  // iteration, by few warps, so its size counts.
  float bound = 0.0f, step = 0.0f, residual = 0.0f;
  std::uint32_t iterations = 0, status = MSB_SOLVE_ITERATION_LIMIT;
  int round = kBound;
#pragma unroll 1
  for (;;) {
    ++comm.round;
    send_sides<P>(d, l, comm, round, step);
    if (round == kFinal) break;
    if (!comm.exchange(l, s)) return kLate;
    Sums x = receive_sides(d, l, round, step);
    if (!reduce(comm, s, x)) return kLate;
    const float value = __uint_as_float(x.bits);
    if (round == kBound) {
      bound = value;
      round = kInitial;
      continue;
    }
    residual = value;
    iterations += round == kIterate ? 1u : 0u;
    if (round == kInitial && (!isfinite(bound) || !(bound > 0.0f))) {
      status = 3;  // no positive diagonal: an invalid system
      round = kFinal;
    } else if (!isfinite(residual)) {
      status = MSB_SOLVE_BREAKDOWN;
      round = kFinal;
    } else if (!(residual > tolerance)) {
      status = MSB_SOLVE_CONVERGED;
      round = kFinal;
    } else {
      step = round == kInitial ? 1.0f / bound : next_step(step, x.v[0], x.v[1], x.v[2], iterations);
      round = iterations < d.max_iterations ? kIterate : kFinal;
    }
  }
  // The solution (the last round wrote its response).
  for (std::uint32_t q = threadIdx.x; q < l.bodies; q += kThreads) {
    const std::uint32_t degree = l.degree(q);
    const std::uint32_t base = base_of(l, q);
    const std::uint32_t begin = d.incidence.offsets[body_at(r, l.first + l.body(q))];
    for (std::uint32_t k = 0; k < degree; ++k) {
      const std::uint32_t side = __float_as_uint(d.incidence.b[begin + k].w);
      if (side & 1u) continue;
      const float4 c = l.c(base + kGroup * k);
      d.multipliers[side >> 1] = c.z;
      d.gaps[side >> 1] = c.w;
      d.iterate[side >> 1] = make_float2(c.z, c.w);
    }
  }
  report = {step, residual, bound, iterations, status};
  return kSolved;
}

// This CTA's inbox and records before its first gang's first word arrives.
__device__ void clear_words(const Comm<kGrid>& comm) {
  const ResidentArrays& r = *comm.arrays;
  unsigned long long* words = r.inbox + std::size_t(comm.first + comm.rank) * r.stride;
  for (std::uint32_t j = threadIdx.x; j < r.stride; j += kThreads) words[j] = 0ull;
  if (threadIdx.x < 2 * kResidentWords) {
    const std::size_t set = std::size_t(threadIdx.x / kResidentWords) * kResidentMaxCtas;
    r.records[(set + comm.first + comm.rank) * kResidentWords + threadIdx.x % kResidentWords] = make_ulonglong2(0ull, 0ull);
  }
  __threadfence();
}

template <int kForm, int P>
__global__ void __launch_bounds__(kThreads, 1)
    resident_kernel(const __grid_constant__ SolveDesc problem, const __grid_constant__ ResidentArrays arrays,
                    SolveDesc* state, std::uint32_t bytes) {
  __shared__ Shared s;
  Comm<kForm> comm{blockIdx.x, gridDim.x, &arrays};
  if constexpr (kForm == kGrid) {
    comm.gang = &state->gang;
    comm.late = &state->gang.late;
    comm.wait_polls = problem.wait_polls;
    clear_words(comm);
  }
  Report report;
  const Outcome outcome = resident_solve<kForm, P>(problem, arrays, comm, s, bytes, 0u, problem.body_count,
                                                   problem.tolerance, &state->check_status, report);
  if constexpr (kForm == kCluster) cg::this_cluster().sync();  // no CTA leaves while another may write its sums
  if (threadIdx.x != 0) return;
  if (outcome == kLate) atomicExch(&state->gang.late, 1u);
  if (comm.rank != 0) return;
  if (outcome == kMisfit) {
    state->gang.misfit = 1u;
  } else if (outcome == kSolved) {
    state->step = report.step;
    state->residual = report.residual;
    state->bound = report.bound;
    state->iterations = report.iterations;
    state->status = report.status;
    state->mode = 1;
  }
}

// A batch: each CTA takes its jobs in order, with the other CTAs of each
// job's gang.  Every list is a part of one sequence of all jobs, so the first
// unfinished job of the sequence always has all of its CTAs.
__global__ void __launch_bounds__(kThreads, 1)
    resident_batch_kernel(const __grid_constant__ SolveDesc problem, const __grid_constant__ ResidentArrays arrays,
                          const __grid_constant__ ResidentBatch batch, std::uint32_t bytes) {
  __shared__ Shared s;
  std::uint32_t round = 0;
  {
    Comm<kGrid> all{blockIdx.x, gridDim.x, &arrays};
    clear_words(all);
  }
  for (std::uint32_t k = batch.list_offsets[blockIdx.x]; k < batch.list_offsets[blockIdx.x + 1]; ++k) {
    const ResidentJob job = batch.jobs[batch.lists[k]];
    const std::uint32_t b0 = batch.cell_offsets[job.colony], b1 = batch.cell_offsets[job.colony + 1];
    const float tolerance = batch.tolerance[job.colony];
    Report report{};
    Outcome outcome;
    std::uint32_t rank = 0;
    if (job.size == 1) {
      Comm<kSingle> comm{0, 1, &arrays};
      outcome = resident_solve<kSingle, 1>(problem, arrays, comm, s, bytes, b0, b1, tolerance, batch.check, report);
    } else {
      Comm<kGrid> comm{blockIdx.x - job.first, job.size,  &arrays, job.first, round, &batch.gangs[batch.lists[k]],
                       batch.late,             problem.wait_polls};
      outcome = resident_solve<kGrid, 1>(problem, arrays, comm, s, bytes, b0, b1, tolerance, batch.check, report);
      rank = comm.rank;
      round = comm.round;
    }
    __syncthreads();
    bool late = outcome == kLate;
    if (threadIdx.x == 0) {
      if (rank == 0) {
        // A colony without rows has no diagonal either, and is converged.
        const bool empty = batch.row_counts[job.colony] == 0u;
        ColonyState& to = batch.state[job.colony];
        if (outcome == kSolved) {
          to = {report.step, empty ? 0.0f : report.residual, report.bound, report.iterations,
                empty ? std::uint32_t(MSB_SOLVE_CONVERGED) : report.status};
        } else {
          to.status = kResidentMisfit;
        }
      }
      if (job.size > 1 && outcome == kSolved && k + 1 < batch.list_offsets[blockIdx.x + 1]) {
        // The others may still read this CTA's last record.
        ResidentGang& gang = batch.gangs[batch.lists[k]];
        __threadfence();
        atomicAdd(&gang.left, 1u);
        late = !wait_count(&gang.left, job.size, problem.wait_polls, batch.late);
      } else if (job.size > 1) {
        atomicAdd(&batch.gangs[batch.lists[k]].left, 1u);
      }
      if (late) atomicExch(batch.late, 1u);
    }
    if (__syncthreads_or(late) != 0) return;
  }
}

// Eight bits of each of x and y, interleaved; both axes at the scale of the
// longer one (the same whatever box scale the search's tuner chose: the order
// decides how a solve's sums are grouped).
__global__ void spatial_keys_kernel(std::uint32_t n, const float4* __restrict__ pos_len, const GridParams* grid_ptr,
                                    const std::uint32_t* __restrict__ colony, std::uint32_t* __restrict__ keys,
                                    std::uint32_t* __restrict__ order) {
  const double x0 = grid_ptr->low[0], y0 = grid_ptr->low[1];
  const double scale = 256.0 / fmax(grid_ptr->span[0], grid_ptr->span[1]);
  for (std::uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float4 p = pos_len[i];
    const auto cell = [&](double at) { return std::uint32_t(fmin(fmax(at * scale, 0.0), 255.0)); };
    const auto spread = [](std::uint32_t v) {
      v = (v | (v << 4)) & 0x0F0Fu;
      v = (v | (v << 2)) & 0x3333u;
      return (v | (v << 1)) & 0x5555u;
    };
    keys[i] = spread(cell(double(p.x) - x0)) | spread(cell(double(p.y) - y0)) << 1 |
              (colony != nullptr ? colony[i] << 16 : 0u);
    order[i] = i;
  }
}

__global__ void order_counts_kernel(std::uint32_t n, const std::uint32_t* __restrict__ order,
                                    const std::uint32_t* __restrict__ offsets, std::uint32_t* __restrict__ counts) {
  for (std::uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i <= n; i += gridDim.x * blockDim.x) {
    const std::uint32_t b = i < n ? order[i] : 0u;
    counts[i] = i < n ? offsets[b + 1] - offsets[b] : 0u;
  }
}

constexpr std::uint32_t kSharedLimit = 227 * 1024;  // of one CTA on an SM
constexpr std::uint32_t kDynamicBytes = (kSharedLimit - std::uint32_t(sizeof(Shared)) - 1024) & ~15u;

template <int kForm, int P>
cudaError_t configure(cudaLaunchConfig_t& config, cudaLaunchAttribute& attribute, int ctas, cudaStream_t stream) {
  const auto kernel = resident_kernel<kForm, P>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kDynamicBytes));
  if (e != cudaSuccess) return e;
  config = cudaLaunchConfig_t{};
  config.gridDim = dim3(unsigned(ctas));
  config.blockDim = dim3(kThreads);
  config.dynamicSmemBytes = kDynamicBytes;
  config.stream = stream;
  config.attrs = &attribute;
  config.numAttrs = kForm == kSingle ? 0 : 1;
  if (kForm == kCluster) {
    // Clusters of 16 CTAs are beyond the portable size of 8.
    if (ctas > 8) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    attribute.id = cudaLaunchAttributeClusterDimension;
    attribute.val.clusterDim.x = unsigned(ctas);
    attribute.val.clusterDim.y = 1;
    attribute.val.clusterDim.z = 1;
  } else if (kForm == kGrid) {
    attribute.id = cudaLaunchAttributeCooperative;
    attribute.val.cooperative = 1;
  }
  return e;
}

template <int kForm, int P>
int launch_form(const SolveDesc& problem, SolveDesc* desc, const ResidentArrays& arrays, int ctas,
                cudaStream_t stream) {
  cudaLaunchConfig_t config;
  cudaLaunchAttribute attribute;
  const cudaError_t e = configure<kForm, P>(config, attribute, ctas, stream);
  if (e != cudaSuccess) return int(e);
  count_launch();
  return int(cudaLaunchKernelEx(&config, resident_kernel<kForm, P>, problem, arrays, desc, kDynamicBytes));
}

template <int kForm>
int launch_lanes(const SolveDesc& problem, SolveDesc* desc, const ResidentArrays& arrays, ResidentPlan plan,
                 cudaStream_t stream) {
  return plan.lanes == 4 ? launch_form<kForm, 4>(problem, desc, arrays, plan.ctas, stream)
                         : launch_form<kForm, 1>(problem, desc, arrays, plan.ctas, stream);
}

}  // namespace

void launch_spatial_order(std::uint32_t n, const float4* pos_len, const GridParams* grid, const std::uint32_t* colony,
                          std::uint32_t colonies, std::uint32_t* keys, std::uint32_t* order, std::uint32_t* temp,
                          cudaStream_t stream) {
  spatial_keys_kernel<<<grid_for(n, 256), 256, 0, stream>>>(n, pos_len, grid, colony, keys, order);
  count_launch();
  radix_sort_pairs(keys, order, n, 16 + (colony != nullptr ? int(std::bit_width(colonies - 1)) : 0), temp, stream);
}

void launch_order_offsets(std::uint32_t n, const std::uint32_t* order, const std::uint32_t* offsets,
                          std::uint32_t* counts, std::uint32_t* order_offsets, std::uint32_t* temp,
                          cudaStream_t stream) {
  order_counts_kernel<<<grid_for(n + 1ull, 256), 256, 0, stream>>>(n, order, offsets, counts);
  count_launch();
  exclusive_scan(counts, order_offsets, n + 1ull, temp, stream);
}

std::uint32_t resident_stride() { return kSharedLimit / kEntryBytes; }

ResidentLimits resident_limits() {
  ResidentLimits limits;
  int device = 0, sms = 0, cooperative = 0, per_sm = 0;
  if (cudaGetDevice(&device) != cudaSuccess) return limits;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  cudaDeviceGetAttribute(&cooperative, cudaDevAttrCooperativeLaunch, device);
  cudaLaunchConfig_t config;
  cudaLaunchAttribute attribute;
  for (const int ctas : {8, 16}) {
    int clusters = 0;
    if (configure<kCluster, 1>(config, attribute, ctas, nullptr) == cudaSuccess &&
        cudaOccupancyMaxActiveClusters(&clusters, resident_kernel<kCluster, 1>, &config) == cudaSuccess && clusters > 0) {
      limits.cluster = ctas;
    }
  }
  if (cooperative != 0 && configure<kGrid, 1>(config, attribute, 1, nullptr) == cudaSuccess &&
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, resident_kernel<kGrid, 1>, kThreads, kDynamicBytes) ==
          cudaSuccess) {
    limits.grid = std::min(sms * per_sm, int(kResidentMaxCtas));
  }
  cudaGetLastError();
  return limits;
}

// What a CTA can hold, less 3 % for the slots that pad the groups of bodies.
constexpr std::uint64_t kShareBytes = std::uint64_t(kDynamicBytes) * 97 / 100;
constexpr std::uint64_t system_bytes(std::uint64_t rows, std::uint64_t bodies) {
  return 2 * rows * kEntryBytes + bodies * kBodyBytes;
}

std::uint32_t resident_ctas(std::uint64_t rows, std::uint64_t bodies) {
  return std::uint32_t(std::min<std::uint64_t>((system_bytes(rows, bodies) + kShareBytes - 1) / kShareBytes, 1u << 30));
}

int launch_resident_batch(const SolveDesc& problem, const ResidentArrays& arrays, const ResidentBatch& batch, int ctas,
                          cudaStream_t stream) {
  cudaError_t e = cudaFuncSetAttribute(resident_batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       int(kDynamicBytes));
  if (e != cudaSuccess) return int(e);
  cudaLaunchConfig_t config{};
  config.gridDim = dim3(unsigned(ctas));
  config.blockDim = dim3(kThreads);
  config.dynamicSmemBytes = kDynamicBytes;
  config.stream = stream;
  cudaLaunchAttribute attribute;
  attribute.id = cudaLaunchAttributeCooperative;
  attribute.val.cooperative = 1;
  config.attrs = &attribute;
  config.numAttrs = 1;
  count_launch();
  return int(cudaLaunchKernelEx(&config, resident_batch_kernel, problem, arrays, batch, kDynamicBytes));
}

ResidentPlan resident_plan(const ResidentLimits& limits, std::uint64_t rows, std::uint64_t bodies) {
  const std::uint64_t bytes = system_bytes(rows, bodies);
  const std::uint64_t share = kShareBytes;
  ResidentPlan plan;
  if (bytes <= share * 3 / 4 || (limits.cluster == 0 && bytes <= share)) {
    plan = {1, false, 1};
  } else if (bytes <= std::uint64_t(limits.cluster) * share) {
    plan = {limits.cluster, false, 1};
  } else if (bytes <= std::uint64_t(limits.grid) * share) {
    plan = {limits.grid, true, 1};
  }
  // Four lanes a body while its CTA's bodies are few; one thread a body keeps
  // more of them in flight.
  if (plan.ctas > 1 && bodies <= 256ull * plan.ctas) plan.lanes = 4;
  return plan;
}

int launch_resident(const SolveDesc& problem, SolveDesc* desc, const ResidentArrays& arrays, ResidentPlan plan,
                    cudaStream_t stream) {
  if (plan.grid) return launch_lanes<kGrid>(problem, desc, arrays, plan, stream);
  if (plan.ctas > 1) return launch_lanes<kCluster>(problem, desc, arrays, plan, stream);
  return launch_form<kSingle, 1>(problem, desc, arrays, plan.ctas, stream);
}

}  // namespace msb
