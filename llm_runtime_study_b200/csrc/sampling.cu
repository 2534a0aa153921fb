// Next-token selection on the device, one thread block per row of logits.
//
// temperature == 0: argmax (the lowest index wins a tie)      mini_llm/sampling.py:80-82
// temperature  > 0: x = logits / temperature; keep the top_k largest; of those keep
//   the smallest set of largest-probability tokens whose mass reaches top_p (a token
//   stays iff the mass of the tokens strictly above it is < top_p, so at least one
//   stays); draw from softmax over what is left              mini_llm/sampling.py:51-69, 87-91
// The draw is Gumbel-max: argmax(x_i + g_i), g_i = -log(-log(u_i)), which samples
// softmax(x) exactly.  u_i comes from a counter-based generator keyed by (request
// seed, index of the token being generated, vocabulary index), so a request's draws
// do not depend on what else is in the batch.  The thresholds for top_k and top_p are found in three
// passes over the row (narrow_threshold): how many elements lie in each of 1,024 (256) equal steps below the
// row's maximum, the same within the steps that can hold the threshold, and the few elements left after that
// exactly; rows of which too many elements are left (equal values, a threshold far below the maximum) by a search over the 32 bits of an
// order-preserving integer key, four bits a pass (find_threshold).  Counts are whole numbers and every sum of weights is taken in an order
// fixed by the launch shape: the same bits every run.
//
// The per-row parameters are six words [temperature bits, top_k, top_p bits, seed low, seed high,
// counter].  They come either as an array [rows][6], or out of the per-request slot records on the
// device (slots.cu): then `row_slots[row]` names the record, and the kernel that settles a row also
// writes the chosen token and the advanced counter back into it, so that the next decode step and
// the next draw need nothing from the host.
#include "common.cuh"
#include "slots.h"

namespace b200 {

constexpr int kParamWords = 6;   // per row: [temperature bits, top_k, top_p bits, seed low, seed high, counter]

// Where a row's six parameter words are, and (slot records only) where its result goes.
struct RowParams {
  int* base;              // [rows][6], or the slot table
  const int* row_slots;   // nullptr: row i uses base + 6 i; else base + kSlotWords * row_slots[i] + kSlotSampling
  __device__ __forceinline__ const int* of(int row) const {
    return row_slots ? base + static_cast<size_t>(row_slots[row]) * kSlotWords + kSlotSampling : base + row * kParamWords;
  }
  // The draw for this row is settled: remember it in the request's record and advance its counter.
  __device__ __forceinline__ void settle(int row, int token, int counter) const {
    if (!row_slots) return;
    int* rec = base + static_cast<size_t>(row_slots[row]) * kSlotWords;
    rec[kSlotLastToken] = token;
    rec[kSlotCounter] = counter + 1;
  }
};

__device__ __forceinline__ uint32_t ordered_key(float x) {
  const uint32_t b = __float_as_uint(x);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

__host__ __device__ __forceinline__ uint64_t splitmix64(uint64_t z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// uniform in (0, 1) from (stream key, vocabulary index): 23 random bits plus one half,
// which float32 holds exactly, so neither 0 nor 1 can come out
__device__ __forceinline__ float uniform23(uint64_t stream, uint32_t index) {
  const uint64_t z = splitmix64(stream + static_cast<uint64_t>(index) * 0xD1B54A32D192ED03ull);
  return (static_cast<float>(static_cast<uint32_t>(z >> 41)) + 0.5f) * (1.0f / 8388608.0f);
}

// A CTA's share of a row: `count` elements from the row's element `base` (a multiple of four) on.
struct Slice {
  const float* x;        // the share: the logits themselves, or the scaled ones staged in shared memory
  int count, base;
  float temperature;     // what x is still to be divided by (1: nothing)
};

// Calls f(scaled logit, vocabulary index) for every element of the slice: 16-byte loads, two in flight per thread,
// then the ragged end.  The order in which a thread sees its elements is fixed by the block size.
template <typename F>
__device__ __forceinline__ void for_each_scaled(const Slice& sl, F&& f) {
  const bool aligned = (reinterpret_cast<uintptr_t>(sl.x) & 15) == 0;
  const int vec = aligned ? sl.count >> 2 : 0;            // whole groups of four
  const float4* x4 = reinterpret_cast<const float4*>(sl.x);
  const int step = blockDim.x;
  const float t = sl.temperature;
  const bool divides = t != 1.f;
  auto four = [&](float4 a, int i) {
    if (divides) { a.x /= t; a.y /= t; a.z /= t; a.w /= t; }
    f(a.x, sl.base + 4 * i);
    f(a.y, sl.base + 4 * i + 1);
    f(a.z, sl.base + 4 * i + 2);
    f(a.w, sl.base + 4 * i + 3);
  };
  int i = threadIdx.x;
  for (; i + step < vec; i += 2 * step) {
    const float4 a = x4[i], b = x4[i + step];
    four(a, i);
    four(b, i + step);
  }
  for (; i < vec; i += step) four(x4[i], i);
  for (int j = 4 * vec + threadIdx.x; j < sl.count; j += step) f(divides ? sl.x[j] / t : sl.x[j], sl.base + j);
}

// ---- reductions over the CTAs of a cluster (a cluster of one is the plain block) ----
// Each CTA puts its block-wide result into a slot of its own shared memory; after a cluster barrier every
// CTA reads the slots of all ranks in rank order, so all of them hold the same bits.  Two sets of slots
// alternate, which makes one barrier per reduction enough.
__device__ __forceinline__ uint32_t cluster_size() {
  uint32_t n;
  asm volatile("mov.u32 %0, %%cluster_nctarank;\n" : "=r"(n));
  return n;
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ float load_from_rank(const float* local, uint32_t rank) {
  uint32_t address = static_cast<uint32_t>(__cvta_generic_to_shared(local)), remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(remote) : "r"(address), "r"(rank));
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v) : "r"(remote) : "memory");
  return v;
}
struct ClusterSlots {
  float (*slots)[16];      // [2][16] in shared memory: what this CTA contributes
  float (*gathered)[16];   // [16 ranks][16]: the contributions of all ranks, fetched by one thread each
  float* totals;           // [16]: their sums
  int which;
};
constexpr int kMaxClusterRanks = 16;
// Sums of the ranks' values, in rank order, into `totals`: every CTA holds the same bits.  slots[which][0 .. n) hold this
// CTA's values and have been written by the threads below `n` of a warp or by one thread; all threads call.
__device__ __forceinline__ void cluster_totals(ClusterSlots& cs, uint32_t ranks, uint32_t n) {
  if (ranks == 1) {
    __syncthreads();
    if (threadIdx.x < n) cs.totals[threadIdx.x] = cs.slots[cs.which][threadIdx.x];
  } else {
    cluster_barrier();
    // one remote load per thread, all in flight together; then a thread per value adds them up
    if (threadIdx.x < ranks * n) cs.gathered[threadIdx.x / n][threadIdx.x % n] = load_from_rank(&cs.slots[cs.which][threadIdx.x % n], threadIdx.x / n);
    __syncthreads();
    if (threadIdx.x < n) {
      float total = 0.f;
      for (uint32_t r = 0; r < ranks; ++r) total += cs.gathered[r][threadIdx.x];
      cs.totals[threadIdx.x] = total;
    }
  }
  __syncthreads();
  cs.which ^= 1;           // two sets of slots alternate: one barrier per reduction is enough
}
__device__ float cluster_sum(float v, float* scratch, ClusterSlots& cs, uint32_t ranks) {
  v = block_sum(v, scratch);
  if (threadIdx.x == 0) cs.slots[cs.which][0] = v;
  cluster_totals(cs, ranks, 1);
  const float total = cs.totals[0];
  __syncthreads();         // read before the next reduction overwrites it
  return total;
}

// Sums of sixteen per-thread values over the block and the cluster, in a fixed order, into cs.totals.  Within a warp each
// exchange halves the values a lane answers for (16 shuffles instead of 5 a value); a warp then finishes one value.
__device__ void sum_sixteen(float (&v)[16], float (*scratch)[32], ClusterSlots& cs, uint32_t ranks) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int o = 16, keep = 8; o > 1; o >>= 1, keep >>= 1) {
    const bool upper = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (i < keep) {
        const float send = upper ? v[i] : v[i + keep];
        v[i] = (upper ? v[i + keep] : v[i]) + __shfl_xor_sync(0xffffffffu, send, o);
      }
    }
  }
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
  if ((lane & 1) == 0) scratch[lane >> 1][warp] = v[0];      // lane 2 n holds value n (its bits chose the halves from the top)
  __syncthreads();
  for (int n = warp; n < 16; n += nwarps) {
    float t = lane < nwarps ? scratch[n][lane] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) cs.slots[cs.which][n] = t;
  }
  cluster_totals(cs, ranks, 16);
}

// The largest key k such that weight(keys >= k) >= target, searched four bits a pass over the whole row
// (every CTA of the cluster scans its slice; the partial weights are added in rank order).  The weight of
// an element is 1 (MASS = false: a count) or exp(v - mx) (MASS = true); elements below `floor_key`
// weigh nothing.  0 when even the whole row does not reach the target.  Elements whose leading bits lie above
// those found so far count in every later pass alike: their weight is carried, and a pass weighs only the
// elements that share the bits found (from the third pass on, few).
template <bool MASS>
__device__ uint32_t find_threshold(const Slice& sl, uint32_t floor_key, float mx, float target, float (*scratch)[32],
                                   ClusterSlots& cs, uint32_t ranks) {
  uint32_t k = 0;
  float above = 0.f;
  for (int shift = 28; shift >= 0; shift -= 4) {
    float w[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) w[j] = 0.f;
    const uint32_t found = shift == 28 ? 0u : k >> (shift + 4);
    for_each_scaled(sl, [&](float v, int) {
      const uint32_t key = ordered_key(v);
      if (key < floor_key || (shift != 28 && (key >> (shift + 4)) != found)) return;
      const uint32_t digit = (key >> shift) & 15u;      // how many of the fifteen candidates the element reaches
      const float weight = MASS ? expf(v - mx) : 1.f;
#pragma unroll
      for (int j = 0; j < 15; ++j)
        if (static_cast<uint32_t>(j) < digit) w[j] += weight;
    });
    sum_sixteen(w, scratch, cs, ranks);
    uint32_t best = 0;
#pragma unroll
    for (int j = 0; j < 15; ++j)
      if (above + cs.totals[j] >= target) best = j + 1;       // weights fall with j: the last one that still reaches the target
    k |= best << shift;
    if (best < 15) above += cs.totals[best];
    __syncthreads();                                          // the totals have been read
  }
  return k;
}

// ---- thresholds in three passes
// An element's place below the maximum is (mx - v) * inv, in steps: a function that never falls as v falls, whatever is rounded, so
// the elements of a step are neighbours in value.  Counts are exact, and the weights of a step's elements are
// known to e^-width, so counts alone say between which steps the threshold lies, for a mass too.
// STEPS: 1,024 for CTAs of 512 threads and more, 256 for smaller ones, whose shares hold fewer elements and whose threads would
// fetch more counts each (256 rows of 32,768 entries, 256 threads: 417 us with 1,024 steps, 162 with 256; 260 before).
constexpr int kLeft = 256;                    // elements that may be left for the end
constexpr float kReach = 32.f;                // the steps reach this far below the maximum (e^-32 of its weight), the last one on from there

template <int STEPS>
struct NarrowMemory {
  int counts[2][STEPS];
  uint32_t left[2][kLeft], gathered[kLeft], sorted[kLeft];   // (left, left_count: a set for each threshold, which other CTAs may still be reading)
  int left_count[2], kept_count, low, high, above;
  float warp_sums[2][32];
  uint32_t result;
  int warp_counts[32];
};

__device__ __forceinline__ uint32_t load_word_from_rank(const void* local, uint32_t rank) {
  uint32_t address = static_cast<uint32_t>(__cvta_generic_to_shared(local)), remote, v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(remote) : "r"(address), "r"(rank));
  asm volatile("ld.shared::cluster.u32 %0, [%1];\n" : "=r"(v) : "r"(remote) : "memory");
  return v;
}
// The word at this place in the first eight ranks' shared memory, all fetched together (0 from ranks that are not there).
constexpr int kRanks = 8;                     // CTAs of a cluster, where there is one
__device__ __forceinline__ void load_from_ranks(const void* local, uint32_t ranks, int (&v)[kRanks]) {
#pragma unroll
  for (int r = 0; r < kRanks; ++r) v[r] = r < static_cast<int>(ranks) ? static_cast<int>(load_word_from_rank(local, r)) : 0;
}
__device__ __forceinline__ float key_value(uint32_t key) { return __uint_as_float((key & 0x80000000u) ? key & 0x7fffffffu : ~key); }

// `sum` becomes the sum of the block-wide sums of all ranks, at the barrier that the counts or the elements left are exchanged behind: a
// meeting of its own would take 2 us.  Two sets of slots alternate, as elsewhere.
__device__ __forceinline__ void meet(float& sum, ClusterSlots& cs, uint32_t ranks) {
  if (ranks == 1) {
    __syncthreads();
    return;
  }
  if (threadIdx.x == 0) cs.slots[cs.which][0] = sum;
  cluster_barrier();
  int v[kRanks];
  load_from_ranks(&cs.slots[cs.which][0], ranks, v);
  sum = 0.f;
#pragma unroll
  for (int r = 0; r < kRanks; ++r) sum += __int_as_float(v[r]);
  cs.which ^= 1;
}

// The steps between which the threshold lies, from the counts of all ranks: with MASS the first that reaches the target if every
// element weighs as much as its step allows, and the first that does if it weighs as little; else the one that reaches it, and the count
// before it.  Step s holds places origin + s * width .. on.  The last step where it is not reached.  MASS: `sum` comes as the
// block-wide sum and goes as the cluster's: the whole weight, `part` of which is the target (FIRST), or the weight of the
// elements before the steps.  All threads call; the counts have been written by atomics of this CTA's threads.
template <bool MASS, bool FIRST, int STEPS>
__device__ void bracket(NarrowMemory<STEPS>& nm, int* counts, ClusterSlots& cs, uint32_t ranks, float origin, float width, float inv, bool open_end,
                        float& sum, float& target, float part, int need) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, each = STEPS / blockDim.x, first = tid * each;
  meet(sum, cs, ranks);
  if (MASS && FIRST) target = part * sum;
  const float before = MASS && !FIRST ? sum : 0.f, slack = FIRST ? 1e-4f : 4e-6f;      // (far beyond what rounding does to the sums)
  const float target_low = target * (1.f - slack), target_high = target * (1.f + slack);
  int mine[8], total = 0;
  float most[8], least[8], sum_most = 0.f, sum_least = 0.f;
  if (tid == 0) { nm.low = nm.high = STEPS - 1; nm.above = 0; }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    mine[i] = 0;
    if (i < each) {
      if (ranks == 1) {
        mine[i] = counts[first + i];
      } else {
        int v[kRanks];
        load_from_ranks(&counts[first + i], ranks, v);
#pragma unroll
        for (int r = 0; r < kRanks; ++r) mine[i] += v[r];
      }
    }
    total += mine[i];
    if (MASS) {
      most[i] = least[i] = 0.f;
      if (mine[i] > 0) {
        const float at = origin + (first + i) * width;      // rounding of places and exponentials: far below 2e-5
        most[i] = mine[i] * expf(-at / inv) * 1.00002f;
        least[i] = open_end && first + i == STEPS - 1 ? 0.f : mine[i] * expf(-(at + width) / inv) * 0.99998f;
      }
      sum_most += most[i];
      sum_least += least[i];
    }
  }
  auto scan = [&](auto v, auto* scratch) {                  // what the threads before this one hold
    auto x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const auto y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) scratch[warp] = x;
    __syncthreads();
    decltype(v) base = 0;
    for (int w = 0; w < warp; ++w) base += scratch[w];
    return base + x - v;
  };
  if (MASS) {
    float upper = before + scan(sum_most, nm.warp_sums[0]), lower = before + scan(sum_least, nm.warp_sums[1]);
    int low = STEPS - 1, high = STEPS - 1;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (i >= each) break;
      upper += most[i];
      lower += least[i];
      if (upper >= target_low) low = min(low, first + i);
      if (lower >= target_high) high = min(high, first + i);
    }
    low = __reduce_min_sync(0xffffffffu, low);
    high = __reduce_min_sync(0xffffffffu, high);
    if (lane == 0) {
      atomicMin(&nm.low, low);
      atomicMin(&nm.high, high);
    }
  } else {
    int count = scan(total, nm.warp_counts);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (i >= each) break;
      if (count < need && count + mine[i] >= need) {
        nm.low = nm.high = first + i;
        nm.above = count;
      }
      count += mine[i];
    }
  }
  __syncthreads();
}

// As find_threshold over the elements whose key is at least floor_key: the largest key k such that weight(keys >= k) reaches
// `need` elements, or `part` of the whole weight (MASS).  ~0u when too many elements are left at the end.
template <bool MASS, int STEPS>
__device__ uint32_t narrow_threshold(const Slice& sl, uint32_t floor_key, float mx, float inv, int need, float part, NarrowMemory<STEPS>& nm,
                                     float* sum_scratch, ClusterSlots& cs, uint32_t ranks) {
  const int tid = threadIdx.x, set = MASS ? 1 : 0;
  auto place = [&](float v) { return fminf((mx - v) * inv, 2.f * STEPS); };
  for (int i = tid; i < STEPS; i += blockDim.x) nm.counts[0][i] = nm.counts[1][i] = 0;
  if (tid == 0) nm.left_count[set] = 0;
  __syncthreads();
  float z = 0.f;
  for_each_scaled(sl, [&](float v, int) {
    if (ordered_key(v) < floor_key) return;
    atomicAdd(&nm.counts[0][min(STEPS - 1, static_cast<int>(place(v)))], 1);
    if (MASS) z += expf(v - mx);
  });
  float target = 0.f;
  if (MASS) z = block_sum(z, sum_scratch);
  bracket<MASS, true, STEPS>(nm, nm.counts[0], cs, ranks, 0.f, 1.f, inv, true, z, target, part, need);
  const int low = nm.low, high = max(nm.high, nm.low), above = nm.above;
  const float finer = static_cast<float>(STEPS) / static_cast<float>(high - low + 1);
  auto fine = [&](float at) { return min(STEPS - 1, static_cast<int>(fminf((at - low) * finer, static_cast<float>(STEPS)))); };
  float m = 0.f;
  for_each_scaled(sl, [&](float v, int) {
    if (ordered_key(v) < floor_key) return;
    const float at = place(v);
    const int step = min(STEPS - 1, static_cast<int>(at));
    if (step < low) {
      if (MASS) m += expf(v - mx);
    } else if (step <= high) {
      atomicAdd(&nm.counts[1][fine(at)], 1);
    }
  });
  float before = MASS ? block_sum(m, sum_scratch) : 0.f;
  bracket<MASS, false, STEPS>(nm, nm.counts[1], cs, ranks, static_cast<float>(low), 1.f / finer, inv, high == STEPS - 1, before, target, part, need - above);
  const int low2 = nm.low, high2 = max(nm.high, nm.low), above2 = nm.above;
  m = 0.f;
  for_each_scaled(sl, [&](float v, int) {
    const uint32_t key = ordered_key(v);
    if (key < floor_key) return;
    const float at = place(v);
    const int step = min(STEPS - 1, static_cast<int>(at));
    if (step < low || step > high) return;
    const int f = fine(at);
    if (f < low2) {
      if (MASS) m += expf(v - mx);
    } else if (f <= high2) {
      const int slot = atomicAdd(&nm.left_count[set], 1);
      if (slot < kLeft) nm.left[set][slot] = key;
    }
  });
  m = MASS ? block_sum(m, sum_scratch) : 0.f;
  meet(m, cs, ranks);
  before += m;
  // every rank's elements, in every CTA; in the order of their keys (those of equal ones does not matter)
  int total = 0, held[kRanks];
  bool fits = true;
  if (ranks == 1) held[0] = nm.left_count[set];
  else load_from_ranks(&nm.left_count[set], ranks, held);
#pragma unroll
  for (int r = 0; r < kRanks; ++r) {
    if (r >= static_cast<int>(ranks)) break;
    fits = fits && held[r] <= kLeft && total + held[r] <= kLeft;
    if (fits)
      for (int i = tid; i < held[r]; i += blockDim.x) nm.gathered[total + i] = ranks == 1 ? nm.left[set][i] : load_word_from_rank(&nm.left[set][i], r);
    total += held[r];
  }
  __syncthreads();
  if (!fits) return ~0u;
  for (int i = tid; i < total; i += blockDim.x) {
    const uint32_t key = nm.gathered[i];
    int rank = 0;
    for (int j = 0; j < total; ++j) rank += nm.gathered[j] > key || (nm.gathered[j] == key && j < i);
    nm.sorted[rank] = key;
  }
  __syncthreads();
  if (tid < 32) {
    uint32_t found = floor_key;
    if (MASS) {
      bool reached = false;
      for (int i0 = 0; i0 < total && !reached; i0 += 32) {      // thirty-two at a time, from the largest on
        found = nm.sorted[min(i0 + tid, total - 1)];
        float mass = i0 + tid < total ? expf(key_value(found) - mx) : 0.f;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const float y = __shfl_up_sync(0xffffffffu, mass, o);
          if (tid >= o) mass += y;
        }
        const unsigned enough = __ballot_sync(0xffffffffu, before + mass >= target);
        before += __shfl_sync(0xffffffffu, mass, 31);
        reached = enough != 0u;
        found = __shfl_sync(0xffffffffu, found, reached ? __ffs(enough) - 1 : 31);
      }
    } else if (total > 0) {
      found = nm.sorted[max(0, min(need - above - above2, total) - 1)];
    }
    if (tid == 0) nm.result = found;
  }
  __syncthreads();
  return nm.result;
}

struct ArgMax {
  float value;
  int index;
};

__device__ __forceinline__ ArgMax better(ArgMax a, ArgMax b) {
  if (b.value > a.value || (b.value == a.value && b.index < a.index)) return b;
  return a;
}

__device__ ArgMax block_argmax(ArgMax v, ArgMax* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgMax other{__shfl_xor_sync(0xffffffffu, v.value, o), __shfl_xor_sync(0xffffffffu, v.index, o)};
    v = better(v, other);
  }
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  const int nwarps = (blockDim.x + 31) >> 5;
  ArgMax t = lane < nwarps ? scratch[lane] : ArgMax{-INFINITY, 0x7fffffff};
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgMax other{__shfl_xor_sync(0xffffffffu, t.value, o), __shfl_xor_sync(0xffffffffu, t.index, o)};
    t = better(t, other);
  }
  return t;  // every thread holds the result
}

// One cluster of CTAs per row (gridDim.x = rows * cluster size): each CTA scans its slice of the row and
// the CTAs combine their results through distributed shared memory.  STAGED: the slice is read from memory and divided by
// the temperature once and kept in shared memory for the passes over it (`staged`: room for it).  32 rows of 151,936 entries, 19 of
// them filtered: 59 us, half of it the passes' arithmetic and half the meetings of the clusters (117 us when each threshold took eight passes of
// find_threshold, which weighs elements against fifteen candidates, and rows without filters two launches of their own); one row with
// top-k 24 us (41), with top-p 40 (52).
template <bool STAGED, int STEPS>
__global__ void __launch_bounds__(1024)
sample_kernel(const float* __restrict__ logits, int ld, int vocab, RowParams params,
              int* __restrict__ out, int filtered_only) {
  __shared__ ArgMax arg_scratch[32];
  __shared__ float sum_scratch[32];
  __shared__ float multi_scratch[16][32];
  __shared__ float slot_memory[2][16];
  __shared__ float gathered_memory[kMaxClusterRanks][16];
  __shared__ float totals[16];
  __shared__ NarrowMemory<STEPS> nm;
  extern __shared__ __align__(16) float staged[];
  pdl_trigger();
  pdl_wait();
  const uint32_t ranks = cluster_size(), rank = cluster_rank();
  const int row = blockIdx.x / ranks;
  const int* p = params.of(row);
  // the whole cluster leaves together: no CTA may wait at a cluster barrier for one that has returned
  if (filtered_only && !(__int_as_float(p[0]) != 0.f && ((p[1] > 0 && p[1] < vocab) || __int_as_float(p[2]) < 1.f))) return;
  const float temperature = __int_as_float(p[0]);
  const int top_k = p[1];
  const float top_p = __int_as_float(p[2]);
  const uint64_t seed = (static_cast<uint64_t>(static_cast<uint32_t>(p[4])) << 32) | static_cast<uint32_t>(p[3]);
  const uint32_t counter = static_cast<uint32_t>(p[5]);
  const int per = ((vocab + static_cast<int>(ranks) - 1) / static_cast<int>(ranks) + 3) & ~3;
  const int begin = min(vocab, static_cast<int>(rank) * per), end = min(vocab, static_cast<int>(rank + 1) * per);
  Slice sl{logits + static_cast<size_t>(row) * ld + begin, end - begin, begin, 1.f};
  ClusterSlots cs{slot_memory, gathered_memory, totals, 0};
  auto cluster_argmax = [&](ArgMax v) {
    v = block_argmax(v, arg_scratch);
    if (ranks == 1) return v;
    if (threadIdx.x == 0) {
      cs.slots[cs.which][0] = v.value;
      cs.slots[cs.which][1] = __int_as_float(v.index);
    }
    cluster_barrier();
    if (threadIdx.x < ranks * 2) {
      const uint32_t r = threadIdx.x >> 1, n = threadIdx.x & 1;
      cs.gathered[r][n] = load_from_rank(&cs.slots[cs.which][n], r);
    }
    __syncthreads();
    ArgMax best{-INFINITY, 0x7fffffff};
    for (uint32_t r = 0; r < ranks; ++r) best = better(best, ArgMax{cs.gathered[r][0], __float_as_int(cs.gathered[r][1])});
    __syncthreads();
    cs.which ^= 1;
    return best;
  };

  // non-finite logits are an error (mini_llm/sampling.py:104-113): report -1
  float bad = 0.f, mx = -INFINITY, mn = INFINITY;
  const float scale = temperature == 0.f ? 1.f : temperature;
  for_each_scaled(sl, [&](float raw, int i) {
    bad += isfinite(raw) ? 0.f : 1.f;
    const float v = raw / scale;
    mx = fmaxf(mx, v);
    mn = fminf(mn, v);
    if (STAGED) staged[i - begin] = v;
  });
  if (STAGED) sl.x = staged;
  else sl.temperature = scale;
  // whether any is not finite, the row's largest and its smallest value, in one exchange (a block-wide barrier: the staged values are there)
  bad = block_sum(bad, sum_scratch);
  mx = block_argmax(ArgMax{mx, 0}, arg_scratch).value;
  mn = -block_argmax(ArgMax{-mn, 0}, arg_scratch).value;
  if (ranks > 1) {
    if (threadIdx.x == 0) {
      cs.slots[cs.which][0] = bad;
      cs.slots[cs.which][1] = mx;
      cs.slots[cs.which][2] = mn;
    }
    cluster_barrier();
    if (threadIdx.x < ranks * 3) cs.gathered[threadIdx.x / 3][threadIdx.x % 3] = load_from_rank(&cs.slots[cs.which][threadIdx.x % 3], threadIdx.x / 3);
    __syncthreads();
    for (uint32_t r = 0; r < ranks; ++r) {
      bad += cs.gathered[r][0];
      mx = fmaxf(mx, cs.gathered[r][1]);
      mn = fminf(mn, cs.gathered[r][2]);
    }
    __syncthreads();
    cs.which ^= 1;
  }
  const bool any_bad = bad > 0.f;
  int result = -1;
  if (!any_bad && temperature == 0.f) {
    ArgMax best{-INFINITY, 0x7fffffff};
    for_each_scaled(sl, [&](float v, int i) { best = better(best, ArgMax{v, i}); });
    result = cluster_argmax(best).index;
  } else if (!any_bad) {
    uint32_t low_key = 0;  // tokens with key >= low_key stay
    const bool cut = top_k > 0 && top_k < vocab;
    if (cut || top_p < 1.f) {
      const bool narrow = isfinite(mx);                      // a tiny temperature may have made infinities of the largest logits
      const float inv = STEPS / fmaxf(fminf(mx - mn, kReach), 1e-20f);
      if (cut) {
        uint32_t key = narrow ? narrow_threshold<false, STEPS>(sl, 0u, mx, inv, top_k, 0.f, nm, sum_scratch, cs, ranks) : ~0u;
        if (key == ~0u) key = find_threshold<false>(sl, 0u, 0.f, static_cast<float>(top_k), multi_scratch, cs, ranks);
        low_key = key;
      }
      if (top_p < 1.f) {
        uint32_t key = narrow ? narrow_threshold<true, STEPS>(sl, low_key, mx, inv, 0, top_p, nm, sum_scratch, cs, ranks) : ~0u;
        if (key == ~0u) {
          float z = 0.f;
          for_each_scaled(sl, [&](float v, int) {
            if (ordered_key(v) >= low_key) z += expf(v - mx);
          });
          const float target = top_p * cluster_sum(z, sum_scratch, cs, ranks);
          key = find_threshold<true>(sl, low_key, mx, target, multi_scratch, cs, ranks);
        }
        low_key = max(low_key, key);
      }
    }
    const uint64_t stream = splitmix64(seed ^ splitmix64(static_cast<uint64_t>(counter)));
    ArgMax best{-INFINITY, 0x7fffffff};
    auto noisy = [&](float v, int i) {
      const float u = uniform23(stream, static_cast<uint32_t>(i));
      best = better(best, ArgMax{v - logf(-logf(u)), i});
    };
    if (low_key == 0u) {
      for_each_scaled(sl, noisy);
    } else {
      // the few that stay are put side by side first: one in a warp would have all of its lanes wait for the noise
      int* kept = &nm.counts[0][0];                          // (the counts have been used)
      constexpr int kKept = 2 * STEPS;
      if (threadIdx.x == 0) nm.kept_count = 0;
      __syncthreads();
      for_each_scaled(sl, [&](float v, int i) {
        if (ordered_key(v) < low_key) return;
        const unsigned together = __activemask();            // the lanes that are here take neighbouring places by one addition
        const int lane = threadIdx.x & 31, first = __ffs(together) - 1;
        int slot = lane == first ? atomicAdd(&nm.kept_count, __popc(together)) : 0;
        slot = __shfl_sync(together, slot, first) + __popc(together & ((1u << lane) - 1u));
        if (slot < kKept) kept[slot] = i;
        else noisy(v, i);
      });
      __syncthreads();
      const int count = min(nm.kept_count, kKept);
      for (int k = threadIdx.x; k < count; k += blockDim.x) {
        const int i = kept[k];
        const float raw = sl.x[i - begin];
        noisy(sl.temperature != 1.f ? raw / sl.temperature : raw, i);
      }
    }
    result = cluster_argmax(best).index;
  }
  // every CTA of the cluster has read the row's parameters by now (the reductions above are barriers)
  if (rank == 0 && threadIdx.x == 0) {
    out[row] = result;
    params.settle(row, result, static_cast<int>(counter));
  }
  if (ranks > 1) cluster_barrier();        // nobody leaves while its slots may still be read
}

// ---------------------------------------------------------------- two-stage selection
// Rows without top_k / top_p need one pass only (argmax of the logits, or of the logits
// plus Gumbel noise), so the vocabulary is cut into `chunks` parts handled by different
// CTAs; the second stage picks the best of the partial results.  Rows with filters take
// the kernel above.
__device__ __forceinline__ bool row_is_filtered(const int* p, int vocab) {
  const float temperature = __int_as_float(p[0]);
  return temperature != 0.f && ((p[1] > 0 && p[1] < vocab) || __int_as_float(p[2]) < 1.f);
}

__global__ void __launch_bounds__(256)
sample_partial_kernel(const float* __restrict__ logits, int ld, int vocab, RowParams params,
                      float* __restrict__ part_value, int* __restrict__ part_index, int chunks) {
  __shared__ ArgMax arg_scratch[32];
  __shared__ float sum_scratch[32];
  pdl_trigger();
  pdl_wait();
  const int row = blockIdx.y, chunk = blockIdx.x;
  const int* p = params.of(row);
  if (row_is_filtered(p, vocab)) return;
  const float* x = logits + static_cast<size_t>(row) * ld;
  const float temperature = __int_as_float(p[0]);
  const uint64_t seed = (static_cast<uint64_t>(static_cast<uint32_t>(p[4])) << 32) | static_cast<uint32_t>(p[3]);
  const uint64_t stream = splitmix64(seed ^ splitmix64(static_cast<uint64_t>(static_cast<uint32_t>(p[5]))));
  const int per = (vocab + chunks - 1) / chunks;
  const int begin = chunk * per, end = min(vocab, begin + per);
  ArgMax best{-INFINITY, 0x7fffffff};
  float bad = 0.f;
  for (int i = begin + threadIdx.x; i < end; i += blockDim.x) {
    const float raw = x[i];
    bad += isfinite(raw) ? 0.f : 1.f;
    float v = raw;
    if (temperature != 0.f) v = raw / temperature - logf(-logf(uniform23(stream, static_cast<uint32_t>(i))));
    best = better(best, ArgMax{v, i});
  }
  best = block_argmax(best, arg_scratch);
  bad = block_sum(bad, sum_scratch);
  if (threadIdx.x == 0) {
    part_value[row * chunks + chunk] = best.value;
    part_index[row * chunks + chunk] = bad > 0.f ? -1 : best.index;
  }
}

__global__ void sample_final_kernel(const float* __restrict__ part_value, const int* __restrict__ part_index,
                                    RowParams params, int vocab, int* __restrict__ out, int chunks) {
  pdl_trigger();
  pdl_wait();
  const int row = blockIdx.x;
  const int* p = params.of(row);
  if (row_is_filtered(p, vocab)) return;   // written by sample_kernel
  const int counter = p[5];
  ArgMax best{-INFINITY, 0x7fffffff};
  bool bad = false;
  for (int c = threadIdx.x; c < chunks; c += 32) {
    const int index = part_index[row * chunks + c];
    if (index < 0) bad = true;
    else best = better(best, ArgMax{part_value[row * chunks + c], index});
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgMax other{__shfl_xor_sync(0xffffffffu, best.value, o), __shfl_xor_sync(0xffffffffu, best.index, o)};
    best = better(best, other);
  }
  bad = __any_sync(0xffffffffu, bad);
  if (threadIdx.x == 0) {
    out[row] = bad ? -1 : best.index;
    params.settle(row, bad ? -1 : best.index, counter);
  }
}

}  // namespace b200

// The single-kernel path: a cluster of eight CTAs per row for vocabularies of 32,768 entries and more, one CTA
// otherwise.  151,936 entries: a share is 76 KB, so two CTAs of 512 threads are resident on an SM and 32 rows run at once.
// Shares of up to 32 KB leave room for more CTAs than 512 threads each do, and rows beyond 64 want them resident at once: 256 threads then.
// 128 rows, all with top-k, 32,768 and 50,257 entries: 77 and 99 us (118 and 149 with 512 threads; 82 and 116 with one CTA a row that reads
// the logits in every pass); 256 rows 137 and 179 us (223 and 283; 162 and 228).  For fewer rows 512 threads are as fast or faster (64 rows, half of
// them filtered: 52 and 66 us against 59 and 80).
constexpr size_t kMostStaged = 200 * 1024, kSmallShare = 32 * 1024;
static int launch_sample(const float* logits, int ld, int vocab, b200::RowParams params, int* out, int rows, int filtered_only,
                         cudaStream_t stream) {
  const int cluster = vocab < 32768 ? 1 : b200::kRanks;
  const size_t share = sizeof(float) * static_cast<size_t>(((vocab + cluster - 1) / cluster + 3) & ~3);
  const int threads = cluster > 1 ? (rows > 64 && share <= kSmallShare ? 256 : 512) : (vocab >= 8192 ? 1024 : (vocab >= 1024 ? 256 : 128));
  const bool staged = share <= kMostStaged;
  auto kernel = threads <= 256 ? (staged ? b200::sample_kernel<true, 256> : b200::sample_kernel<false, 256>)
                               : (staged ? b200::sample_kernel<true, 1024> : b200::sample_kernel<false, 1024>);
  static b200::DeviceOnce once[2];
  if (staged)
    if (int e = b200::configure_once(once[threads > 256], kernel, kMostStaged)) return e;
  cudaLaunchConfig_t config{};
  config.gridDim = dim3(rows * cluster);
  config.blockDim = dim3(threads);
  config.dynamicSmemBytes = staged ? share : 0;
  config.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attr;
  config.numAttrs = b200::pdl_enabled() ? 2 : 1;
  cudaError_t e = cudaLaunchKernelEx(&config, kernel, logits, ld, vocab, params, out, filtered_only);
  return static_cast<int>(e != cudaSuccess ? e : cudaGetLastError());
}

extern "C" int b200_sample(const float* logits, int ld, int vocab, const int* params, int* out,
                           int rows, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (vocab <= 0 || ld < vocab) return B200_ERR_BAD_SIZE;
  return launch_sample(logits, ld, vocab, b200::RowParams{const_cast<int*>(params), nullptr}, out, rows, 0, stream);
}

// Up to so many rows, if some are filtered, all of them in the one launch: the rows without filters beside the others (32 rows of 151,936 entries: the
// two launches before it took 17 us).
constexpr int kRowsTogether = 64;

// Two-stage variant.  `scratch` holds rows * chunks floats followed by rows * chunks ints;
// `any_filtered` tells whether some row uses top_k / top_p (then the kernel with a cluster per row
// also runs, for those rows only).
static int sample_chunked(const float* logits, int ld, int vocab, b200::RowParams params, int* out, int rows,
                          int chunks, void* scratch, int any_filtered, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (vocab <= 0 || ld < vocab || chunks <= 0 || rows > 65535) return B200_ERR_BAD_SIZE;
  if (any_filtered && rows <= kRowsTogether) return launch_sample(logits, ld, vocab, params, out, rows, 0, stream);
  float* part_value = static_cast<float*>(scratch);
  int* part_index = reinterpret_cast<int*>(part_value + static_cast<size_t>(rows) * chunks);
  dim3 grid(chunks, rows);
  b200::launch(b200::sample_partial_kernel, dim3(grid), dim3(256), 0, stream, logits, ld, vocab, params, part_value, part_index, chunks);
  b200::launch(b200::sample_final_kernel, dim3(rows), dim3(32), 0, stream, part_value, part_index, params, vocab, out, chunks);
  if (int e = b200::launch_status()) return e;
  if (any_filtered) return launch_sample(logits, ld, vocab, params, out, rows, 1, stream);
  return 0;
}

extern "C" int b200_sample_chunked(const float* logits, int ld, int vocab, const int* params, int* out, int rows,
                                   int chunks, void* scratch, int any_filtered, cudaStream_t stream) {
  return sample_chunked(logits, ld, vocab, b200::RowParams{const_cast<int*>(params), nullptr}, out, rows, chunks, scratch,
                        any_filtered, stream);
}

// The same selection with the rows' parameters taken from the slot records (`records`: the table,
// `row_slots[i]`: the record of row i): the chosen token and the advanced counter are written back
// into the record as well as into `out`.
extern "C" int b200_sample_slots(const float* logits, int ld, int vocab, int* records, const int* row_slots, int* out,
                                 int rows, int chunks, void* scratch, int any_filtered, cudaStream_t stream) {
  if (records == nullptr || row_slots == nullptr) return B200_ERR_BAD_SIZE;
  return sample_chunked(logits, ld, vocab, b200::RowParams{records, row_slots}, out, rows, chunks, scratch, any_filtered, stream);
}
