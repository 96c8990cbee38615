// Sampling on the device, one team of thread blocks per row of 32-bit logits.
//
// What the reference's sampler computes (crates/xrt-runtime/src/sampler.rs):
//   repetition penalty p > 1 on every id seen in the history: l > 0 ? l / p : l * p      :77-91, 110-125
//   temperature <= 1e-5: argmax, the first maximum wins                                    :63, 83-98
//   else: keep the top_k largest adjusted logits (0 = all)                                 :107-145
//         probabilities exp((l - max) / T), normalised                                     :148-164
//         keep the shortest prefix, by falling probability, whose sum reaches top_p        :166-183
//         draw r in [0, 1) and walk the cumulative sum                                     :186-195
// The reference sorts the candidates; here nothing is sorted.  A radix select over order-preserving
// keys finds the top_k threshold (by count) and the top_p threshold (by probability mass), equal
// values at a threshold are kept in index order (the reference's heap also keeps the earlier of
// equal values), and the draw walks the kept set in index order.  The kept set and its
// probabilities are those of the reference; which id a given r lands on is this library's own
// convention, as is the generator: u = top 32 bits of
// splitmix64(key[slot] + (counter[slot] + 1) * 0x9E3779B97F4A7C15), counter[slot] += 1 a draw.
// Probability mass is summed as 64-bit integers (probability * 2^32), so sums do not depend on
// the order in which threads add and a seed gives the same tokens on every run.
//
// A row is worked on by a team of up to eight blocks (one thread-block cluster), each with a contiguous slice of the
// vocabulary: a row of 128,256 logits is half a megabyte, and one block alone was bound by the latency of its passes over it.
// A block reads its slice once, applies the penalty and keeps the values in shared memory.  A small top_k leaves few
// candidates, which the first block finishes by itself; without one, the team goes through the
// selects together, meeting once a pass.
// Measured, microseconds, one block a row -> teams: 128,256 logits, top_k 40, top_p 0.95, 1 row 136 -> 21, 64 rows 145 -> 57; top_p
// 0.9 alone 559 -> 62 and 571 -> 169; greedy 32 -> 6 and 34 -> 14; top_k 500 136 -> 33 and 151 -> 91.  Memory would take 5 for 64 rows.
// One row is a chain of latencies: the pass over the slice, the team's meetings, the ranking.  64 rows of that kernel run it twice, since
// two blocks fill a multiprocessor (64 registers a thread of 512; 85 KB) and there are 512.
//
// Batches that would take two rounds and whose rows all have a small top_k (the usual options; the caller says so) or are greedy take
// the SMALL form: no values kept, so that four blocks of 32,064 logits a row run all at once, and one cut for the whole team, so that hardly more
// than top_k candidates remain and only the threads that hold one look at the logits again.  64 rows of 128,256, top_k 40, top_p 0.95,
// the kernel alone, values kept -> SMALL: normal logits 63 -> 27 us; all rows masked to 11 ids 192 -> 25, with the lowest number for a mask 199 -> 37,
// in falling order 171 -> 42, of one value 212 -> 31; one such row among them 78 -> 27, 81 -> 32, 72 -> 35, 84 -> 28.  Of fewer rows the values
// are worth their place (16 rows of 32,000: 18.9, SMALL with eight blocks a row 27.3).
#include <type_traits>

#include "common.cuh"

namespace xrt {

constexpr int SAMPLE_THREADS = 512, SAMPLE_WARPS = SAMPLE_THREADS / 32;
constexpr int SAMPLE_TEAM = 8;                             // blocks of a team at most
constexpr int SAMPLE_HIST_COPIES = SAMPLE_THREADS / 64;    // private histograms of the radix select
constexpr int SAMPLE_FINE_BINS = 4096;                     // of the first histogram: the order key's top 12 bits
constexpr int SAMPLE_HIST_BYTES = SAMPLE_FINE_BINS * 4;    // also room for the private histograms, and for a block's candidates
constexpr int SAMPLE_CANDIDATES = 4096;                    // of a small top_k, all blocks together
constexpr int SAMPLE_NARROW = 192;                         // so many candidates are cut down once more
constexpr int SAMPLE_CACHED_BYTES = 160 * 1024;            // of logits a block keeps at most
constexpr int SAMPLE_GROUPS = SAMPLE_THREADS / 8;          // of a block in the SMALL form: eight lanes each
constexpr uint32_t SAMPLE_LOWEST_KEY = 0x007fffffu;        // the order key of minus infinity
static_assert(SAMPLE_HIST_COPIES * 256 * 8 <= SAMPLE_HIST_BYTES && SAMPLE_CANDIDATES * 8 <= 32 * 1024, "the regions hold");

__device__ __forceinline__ uint64_t sm64(uint64_t x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

// larger float <=> larger key; NaN sorts lowest
__device__ __forceinline__ uint32_t order_key(float v) {
  if (v != v) return 0u;
  const uint32_t b = __float_as_uint(v);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

struct RowView {
  const float* logits;
  const uint32_t* seen;  // bitmap of ids in the history, or null
  float penalty;
  __device__ __forceinline__ float adjusted(int i) const {
    float l = logits[i];
    if (seen != nullptr && ((seen[i >> 5] >> (i & 31)) & 1u)) l = l > 0.f ? l / penalty : l * penalty;
    return l;
  }
};

__device__ __forceinline__ uint64_t shfl_up64(uint64_t v, int delta) {
  const uint32_t lo = __shfl_up_sync(0xffffffffu, (uint32_t)v, delta);
  const uint32_t hi = __shfl_up_sync(0xffffffffu, (uint32_t)(v >> 32), delta);
  return ((uint64_t)hi << 32) | lo;
}

// Exclusive prefix sum of one value a thread over the block, in thread order; *total gets the sum.
__device__ uint64_t block_exclusive_scan(uint64_t v, uint64_t* warp_totals, uint64_t* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint64_t inc = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint64_t up = shfl_up64(inc, d);
    if (lane >= d) inc += up;
  }
  __syncthreads();
  if (lane == 31) warp_totals[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    uint64_t w = lane < (blockDim.x >> 5) ? warp_totals[lane] : 0;
    uint64_t winc = w;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint64_t up = shfl_up64(winc, d);
      if (lane >= d) winc += up;
    }
    warp_totals[lane] = winc - w;          // exclusive offsets of the warps
    if (lane == 31) warp_totals[32] = winc;  // grand total
  }
  __syncthreads();
  *total = warp_totals[32];
  return warp_totals[warp] + inc - v;
}

// ------------------------------------------------------------------------------------------ the team
__device__ __forceinline__ void team_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void team_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ void team_sync() { team_arrive(); team_wait(); }
// The same variable in the shared memory of block `rank` of the team.
template <typename T>
__device__ __forceinline__ T* of_block(T* p, int rank) {
  uint64_t mapped;
  asm("mapa.u64 %0, %1, %2;" : "=l"(mapped) : "l"(reinterpret_cast<uint64_t>(p)), "r"(rank));
  return reinterpret_cast<T*>(mapped);
}

struct SampleShared {
  uint64_t scan[33];
  uint64_t exchange[2][SAMPLE_TEAM];   // a number from every block, two meetings in turn
  uint64_t best[SAMPLE_TEAM];          // every block's largest value and where
  unsigned long long merged[2][256];   // this block's histogram of a pass, two passes in turn
  uint64_t selected_inside, selected_at;
  uint32_t selected_prefix;
  int selected;
  int count;                           // this block's candidates, -1: too many
  int cut;
  unsigned int draw;
  long long pick;
  int warp_count[SAMPLE_WARPS];
};

// What the SMALL form has beside: the largest order keys of every group of every block, the cut, and the first block's candidates.
struct SmallShared {
  alignas(16) uint32_t group_key[SAMPLE_TEAM * SAMPLE_GROUPS];
  uint32_t own_key[SAMPLE_GROUPS];
  uint32_t cut;
  int count;
  int ties[SAMPLE_TEAM];  // of every block
  int id[SAMPLE_CANDIDATES];
  float value[SAMPLE_CANDIDATES];
};

struct Team {
  SampleShared* sh;
  uint32_t* hist;  // SAMPLE_HIST_BYTES
  int size, rank, turn;
};

// Exclusive prefix sum of one value a thread over the team, blocks in rank order, threads in thread order; *total gets the sum.
template <bool TEAM>
__device__ uint64_t team_exclusive_scan(uint64_t v, Team& team, uint64_t* total) {
  uint64_t before = block_exclusive_scan(v, team.sh->scan, total);
  if (TEAM) {
    uint64_t* mine = team.sh->exchange[team.turn];
    team.turn ^= 1;
    if ((int)threadIdx.x < team.size) of_block(mine, threadIdx.x)[team.rank] = *total;
    team_sync();
    uint64_t sum = 0;
    for (int r = 0; r < team.size; ++r) {
      if (r == team.rank) before += sum;
      sum += mine[r];
    }
    *total = sum;
  }
  return before;
}

// The first place, in index order, at which the running sum of weight(i) exceeds `target`; -1 if the whole sum does not.
// Places of a block's elements count from `base`.  A warp owns a contiguous run of elements, its lanes side by side.
template <bool TEAM, typename F>
__device__ long long ordered_pick(F weight, int n, int base, uint64_t target, Team& team) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int run = ((n + SAMPLE_WARPS - 1) / SAMPLE_WARPS + 31) & ~31;
  const int lo = min(n, warp * run), hi = min(n, lo + run);
  uint64_t local = 0;
  for (int i = lo + lane; i < hi; i += 32) local += weight(i);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(0xffffffffu, (unsigned long long)local, o);
  if (threadIdx.x == 0) team.sh->pick = -1;
  uint64_t total;
  uint64_t before = team_exclusive_scan<TEAM>(lane == 0 ? local : 0, team, &total);
  before = __shfl_sync(0xffffffffu, (unsigned long long)before, 0);
  if (before <= target && target < before + local) {  // one warp of the team
    for (int i0 = lo; i0 < hi; i0 += 32) {
      const int i = i0 + lane;
      uint64_t inc = i < hi ? weight(i) : 0;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint64_t up = shfl_up64(inc, d);
        if (lane >= d) inc += up;
      }
      const unsigned reached = __ballot_sync(0xffffffffu, before + inc > target);
      if (reached) {
        const long long place = (long long)base + i0 + (__ffs(reached) - 1);
        if (TEAM) {
          if (lane < team.size) *of_block(&team.sh->pick, lane) = place;
        } else if (lane == 0) {
          team.sh->pick = place;
        }
        break;
      }
      before += __shfl_sync(0xffffffffu, (unsigned long long)inc, 31);
    }
  }
  if (TEAM) team_sync();
  else __syncthreads();
  const long long found = team.sh->pick;
  __syncthreads();  // the next call resets it
  return found;
}

// The mass of a value: 2^32 times its probability over the largest value's, rounded down.  None for a NaN, and none for an
// infinity against another (the row's first infinity is then its id, as the first maximum without any mass).
__device__ __forceinline__ uint64_t probability_mass(float a, float row_max, float inv_temp) {
  return (uint64_t)(fmaxf(expf((a - row_max) * inv_temp), 0.f) * 4294967296.0f);  // (the larger of a NaN and 0 is 0)
}

// Radix select from the top: the largest key K such that the weight of {key >= K} reaches `want` (>= 1).
// Returns the key; *inside gets want minus the weight of {key > K} (what the keys equal to K still
// have to supply) and *at_key the weight of {key == K}.  If the whole weight is below `want`, returns 0 with *inside = 0.
// weight <= 2^32.  `wide`: so many elements that a bin's sum of 16-bit halves could pass 32 bits.
// each(f): f(i, value) for every element of this thread, in any order.
template <bool TEAM, typename E, typename F>
__device__ uint32_t radix_select(E each, F weight, uint64_t want, bool wide, Team& team, uint64_t* inside, uint64_t* at_key) {
  SampleShared* sh = team.sh;
  uint32_t prefix = 0, mask = 0;
  uint64_t remaining = want;
  for (int pass = 3; pass >= 0; --pass) {
    const int shift = pass * 8;
    // private histograms (a pair of warps shares one): logits crowd into a few bins of the leading byte.  A bin is two
    // 32-bit sums, of the weights' low and high 16 bits: adding 64 bits to shared memory is a compare-and-swap loop.
    uint32_t* mine = team.hist + (threadIdx.x >> 6) * 512;
    for (int b = threadIdx.x; b < SAMPLE_HIST_COPIES * 512; b += SAMPLE_THREADS) team.hist[b] = 0u;
    if (threadIdx.x == 0) sh->selected = 0;
    __syncthreads();
    each([&](int i, float a) {
      const uint32_t k = order_key(a);
      if ((k & mask) == prefix) {
        const uint64_t w = weight(i, a);
        const uint32_t bin = (k >> shift) & 255u;
        if (wide) {
          if (w) atomicAdd(reinterpret_cast<unsigned long long*>(mine) + bin, (unsigned long long)w);
        } else {
          const uint32_t low = (uint32_t)w & 0xffffu, high = (uint32_t)(w >> 16);
          if (low) atomicAdd(&mine[2 * bin], low);
          if (high) atomicAdd(&mine[2 * bin + 1], high);
        }
      }
    });
    __syncthreads();
    unsigned long long* merged = sh->merged[pass & 1];
    unsigned long long sum = 0ull;
    const int bin = 255 - (int)threadIdx.x;  // from the top
    if (bin >= 0) {
#pragma unroll
      for (int c = 0; c < SAMPLE_HIST_COPIES; ++c) {
        if (wide) sum += reinterpret_cast<unsigned long long*>(team.hist)[c * 256 + bin];
        else sum += (unsigned long long)team.hist[c * 512 + 2 * bin] + ((unsigned long long)team.hist[c * 512 + 2 * bin + 1] << 16);
      }
    }
    if (TEAM) {
      if (bin >= 0) merged[bin] = sum;
      team_sync();
      sum = 0ull;
      if (bin >= 0)
        for (int r = 0; r < team.size; ++r) sum += of_block(merged, r)[bin];
    }
    uint64_t total;
    const uint64_t above = block_exclusive_scan(sum, sh->scan, &total);
    if (above < remaining && remaining <= above + sum) {  // one thread, unless there is not enough weight in all
      sh->selected = 1;
      sh->selected_prefix = prefix | ((uint32_t)bin << shift);
      sh->selected_inside = remaining - above;
      sh->selected_at = sum;
    }
    __syncthreads();
    if (!sh->selected) {
      *inside = 0; *at_key = 0;
      __syncthreads();
      return 0u;
    }
    prefix = sh->selected_prefix;
    mask |= 255u << shift;
    remaining = sh->selected_inside;
    *at_key = sh->selected_at;
    __syncthreads();
  }
  *inside = remaining;
  return prefix;
}

// From the values to the id: top_k, top_p and the draw over `n` elements of this block, whose places count from `base`.
// TEAM: over the elements of all blocks.  adjusted(i): element i; each(f): see radix_select.  Returns the place of the id, -1 if no
// mass was left.
template <bool TEAM, typename A, typename E>
__device__ long long sample_place(A adjusted, E each, int n, int base, long long n_all, int k, float temp, float p, float row_max,
                                  bool wide, Team& team) {
  // top-k: threshold key and the last place kept among equal keys
  uint32_t k_key = 0u; long long k_last = n_all;  // kept: key > k_key, or key == k_key and place <= k_last
  if (k > 0 && k < n_all) {
    uint64_t inside, at_key;
    auto one = [&](int, float) { return (uint64_t)1; };
    k_key = radix_select<TEAM>(each, one, (uint64_t)k, wide, team, &inside, &at_key);
    if (at_key > inside) {
      auto tie = [&](int i) { return (uint64_t)(order_key(adjusted(i)) == k_key); };
      k_last = ordered_pick<TEAM>(tie, n, base, inside - 1, team);
    }
  }
  const float inv_temp = 1.0f / temp;
  auto mass_of = [&](int i, float a) -> uint64_t {
    const uint32_t key = order_key(a);
    if (key < k_key || (key == k_key && base + i > k_last)) return 0ull;
    return probability_mass(a, row_max, inv_temp);
  };
  // top-p: threshold by probability mass
  uint32_t p_key = 0u; long long p_last = n_all;
  if (p < 1.0f) {
    uint64_t local = 0, total;
    each([&](int i, float a) { local += mass_of(i, a); });
    team_exclusive_scan<TEAM>(local, team, &total);
    uint64_t want = (uint64_t)ceil((double)p * (double)total);
    if (want < 1) want = 1;
    uint64_t inside, at_key;
    p_key = radix_select<TEAM>(each, mass_of, want, wide, team, &inside, &at_key);
    if (at_key > inside) {
      // equal keys have equal mass: how many of them the remaining mass needs
      auto tie_mass = [&](int i) { const float a = adjusted(i); return order_key(a) == p_key ? mass_of(i, a) : 0ull; };
      p_last = ordered_pick<TEAM>(tie_mass, n, base, inside - 1, team);
    }
  }
  auto kept_of = [&](int i, float a) -> uint64_t {
    const uint32_t key = order_key(a);
    if (key < p_key || (key == p_key && base + i > p_last)) return 0ull;
    return mass_of(i, a);
  };
  auto kept_mass = [&](int i) { return kept_of(i, adjusted(i)); };
  uint64_t local = 0, total;
  each([&](int i, float a) { local += kept_of(i, a); });
  team_exclusive_scan<TEAM>(local, team, &total);
  const uint64_t target = __umul64hi((uint64_t)team.sh->draw << 32, total);  // floor(u / 2^32 * total)
  return total > 0 ? ordered_pick<TEAM>(kept_mass, n, base, target, team) : -1;
}

// `hist` holds, by the top 12 bits of their order keys, numbers that say: at least so many elements lie in this bin; TEAM: the
// numbers of all blocks together.  The bin at which they reach k from the top, 0 if they don't.
template <bool TEAM>
__device__ uint32_t find_cut(uint32_t* hist, int k, Team& team) {
  const int blocks = TEAM ? team.size : 1;
  const int bins = SAMPLE_FINE_BINS / (SAMPLE_THREADS * blocks);  // of a thread: the first block's first has the top ones
  const int first = SAMPLE_FINE_BINS - bins * ((TEAM ? team.rank * SAMPLE_THREADS : 0) + (int)threadIdx.x + 1);
  auto bin = [&](int i) {
    uint32_t sum = 0;
    for (int r = 0; r < blocks; ++r) sum += (TEAM ? of_block(hist, r) : hist)[i];
    return sum;
  };
  uint64_t local = 0, total;
  if (threadIdx.x == 0) team.sh->cut = 0;
  for (int i = first; i < first + bins; ++i) local += bin(i);
  uint64_t above = team_exclusive_scan<TEAM>(local, team, &total);
  if (above < (uint64_t)k && (uint64_t)k <= above + local) {  // one thread
    int cut = first + bins;
    while (above < (uint64_t)k) above += bin(--cut);
    for (int r = 0; r < blocks; ++r) *(TEAM ? of_block(&team.sh->cut, r) : &team.sh->cut) = cut;
  }
  if (TEAM) team_sync();  // (also: everybody is done with the others' histograms)
  else __syncthreads();
  return (uint32_t)team.sh->cut;
}

// Copies every element whose order key's top 12 bits are `cut` or more to out_id / out_val, in index order, if there are no
// more than `cap`.  Returns how many there are.  The outputs may be the histogram's own room.
template <typename A, typename I>
__device__ int gather(A adjusted, I id_of, int n, uint32_t cut, int cap, SampleShared* sh, int* out_id, float* out_val) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (cut == 0 && n > cap) return n;
  const int run = ((n + SAMPLE_WARPS - 1) / SAMPLE_WARPS + 31) & ~31;
  const int lo = min(n, warp * run), hi = min(n, lo + run);
  int mine = 0;
  for (int i0 = lo; i0 < hi; i0 += 32) {
    const int i = i0 + lane;
    mine += __popc(__ballot_sync(0xffffffffu, i < hi && (order_key(adjusted(i)) >> 20) >= cut));
  }
  if (lane == 0) sh->warp_count[warp] = mine;
  __syncthreads();  // also: everybody is done with the histogram
  int at = 0, count = 0;
  for (int w = 0; w < SAMPLE_WARPS; ++w) {
    if (w == warp) at = count;
    count += sh->warp_count[w];
  }
  if (count <= cap) {
    for (int i0 = lo; i0 < hi && mine > 0; i0 += 32) {
      const int i = i0 + lane;
      const float a = i < hi ? adjusted(i) : 0.f;
      const bool in = i < hi && (order_key(a) >> 20) >= cut;
      const unsigned mask = __ballot_sync(0xffffffffu, in);
      if (in) {
        const int place = at + __popc(mask & ((1u << lane) - 1u));
        out_id[place] = id_of(i);
        out_val[place] = a;
      }
      at += __popc(mask);
    }
  }
  __syncthreads();
  return count;
}

// The same choice as sample_place over no more candidates than threads, each thread its own: its rank is the number of
// candidates before it by falling value (equal values in index order), the mass before it theirs.  `order` and `mass`:
// shared memory for SAMPLE_THREADS numbers each.
__device__ long long ranked_place(float a, int n, int k, float temp, float p, float row_max, uint64_t* order, uint64_t* mass,
                                  Team& team) {
  const int i = threadIdx.x;
  const uint64_t mine = ((uint64_t)order_key(a) << 32) | (uint32_t)~(uint32_t)i;
  if (i < n) order[i] = mine;
  if (i == 0) team.sh->pick = -1;
  __syncthreads();
  int rank = n;
  if ((i & ~31) < n) {
    rank = 0;
#pragma unroll 4
    for (int j = 0; j < n; ++j) rank += order[j] > mine;
  }
  const uint64_t m = i < n && rank < k ? probability_mass(a, row_max, 1.0f / temp) : 0ull;
  if (i < n) mass[i] = m;
  uint64_t total;
  block_exclusive_scan(m, team.sh->scan, &total);
  uint64_t kept = m;
  if (p < 1.0f) {
    uint64_t want = (uint64_t)ceil((double)p * (double)total);
    if (want < 1) want = 1;
    uint64_t before = 0;
    if (__any_sync(0xffffffffu, m != 0)) {
#pragma unroll 4
      for (int j = 0; j < n; ++j) before += order[j] > mine ? mass[j] : 0ull;
    }
    if (before >= want) kept = 0;
  }
  const uint64_t below = block_exclusive_scan(kept, team.sh->scan, &total);
  const uint64_t target = __umul64hi((uint64_t)team.sh->draw << 32, total);  // floor(u / 2^32 * total)
  if (total > 0 && below <= target && target < below + kept) team.sh->pick = i;
  __syncthreads();
  return team.sh->pick;
}

// The same choice for candidates in any order (ids[i], vals[i], no more than threads, all of the row's values at or above its
// k-th largest among them): places are compared by id.  Returns the id.  `order`, `mass`: shared memory for SAMPLE_THREADS numbers each.
__device__ int ranked_id(const int* ids, const float* vals, int n, int k, float temp, float p, float row_max, int row_arg,
                         uint64_t* order, uint64_t* mass, Team& team) {
  const int i = threadIdx.x;
  const bool live = i < n, warp_live = (i & ~31) < n;
  const int id = live ? ids[i] : 0;
  const float a = live ? vals[i] : 0.f;
  const uint64_t mine = ((uint64_t)order_key(a) << 32) | (uint32_t)~(uint32_t)id;
  if (live) order[i] = mine;
  if (i == 0) team.sh->pick = -1;
  __syncthreads();
  int rank = n;
  if (warp_live) {
    rank = 0;
#pragma unroll 4
    for (int j = 0; j < n; ++j) rank += order[j] > mine;
  }
  const uint64_t m = live && rank < k ? probability_mass(a, row_max, 1.0f / temp) : 0ull;
  if (live) mass[i] = m;
  uint64_t total;
  block_exclusive_scan(m, team.sh->scan, &total);
  uint64_t kept = m;
  if (p < 1.0f) {
    uint64_t want = (uint64_t)ceil((double)p * (double)total);
    if (want < 1) want = 1;
    uint64_t before = 0;
    if (warp_live) {
#pragma unroll 4
      for (int j = 0; j < n; ++j) before += order[j] > mine ? mass[j] : 0ull;
    }
    if (before >= want) kept = 0;
    __syncthreads();  // the masses are read: what is kept of them takes their place
    if (live) mass[i] = kept;
  }
  block_exclusive_scan(kept, team.sh->scan, &total);  // (its barriers: the kept masses are there)
  uint64_t below = 0;
  if (warp_live) {
    const uint32_t place = (uint32_t)mine;  // falls as the id rises
#pragma unroll 4
    for (int j = 0; j < n; ++j) below += (uint32_t)order[j] > place ? mass[j] : 0ull;
  }
  const uint64_t target = __umul64hi((uint64_t)team.sh->draw << 32, total);  // floor(u / 2^32 * total)
  if (total > 0 && below <= target && target < below + kept) team.sh->pick = id;
  __syncthreads();
  return team.sh->pick >= 0 ? (int)team.sh->pick : row_arg;
}

// Lists the first `want` places, in index order over the team's blocks, where tie(i) holds, behind the first `at` entries of the
// first block's candidates.  `ties`: every block's count, in every block.  Returns whether so many places hold.  Ends with a meeting.
template <typename P, typename A>
__device__ bool send_ties(P tie, A adjusted, int n, int base, int want, SmallShared* first, int at, int* warp_count, int* ties,
                          Team& team) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int run = ((n + SAMPLE_WARPS - 1) / SAMPLE_WARPS + 31) & ~31;
  const int lo = min(n, warp * run), hi = min(n, lo + run);
  int mine = 0;  // (counted no further than matters)
  for (int i0 = lo; i0 < hi && mine < want; i0 += 32) mine += __popc(__ballot_sync(0xffffffffu, i0 + lane < hi && tie(i0 + lane)));
  if (lane == 0) warp_count[warp] = mine;
  __syncthreads();
  int place = 0, all = 0;
  for (int w = 0; w < SAMPLE_WARPS; ++w) {
    if (w < warp) place += warp_count[w];
    all += warp_count[w];
  }
  if ((int)threadIdx.x < team.size) of_block(ties, threadIdx.x)[team.rank] = all;
  team_sync();
  all = 0;
  for (int r = 0; r < team.size; ++r) {
    if (r < team.rank) place += ties[r];
    all += ties[r];
  }
  for (int i0 = lo; i0 < hi && place < want; i0 += 32) {
    const int i = i0 + lane;
    const bool in = i < hi && tie(i);
    const unsigned mask = __ballot_sync(0xffffffffu, in);
    const int here = place + __popc(mask & ((1u << lane) - 1u));
    if (in && here < want) {
      first->id[at + here] = base + i;
      first->value[at + here] = adjusted(i);
    }
    place += __popc(mask);
  }
  team_sync();
  return all >= want;
}

// CACHED: a block's slice of the row fits its shared memory (else the passes read it from the L2 again).
// VEC: rows are whole 16 bytes.
// SMALL (not CACHED): for batches whose rows have a small top_k or are greedy.  The row's cut is the k-th largest of the largest values
// of all groups of eight lanes of the team (64 a block): k values lie at or above it, and with twice as many groups as k hardly more.
// Every block gets every group's value (one meeting) and finds the cut by itself; a thread whose own largest value reaches it
// looks at its logits again and lists what lies at or above the cut in the first block, which ranks the candidates.  Where more than
// that is at the cut (rows masked with a lowest value, or whose values are equal), what lies above it is listed, and the first of its equals; more
// than are ranked at once are cut once more.  A row that this does not serve (a larger k, thousands above the cut, too many in the bin
// of the second one, a cut at zero with too few zeros without a sign) goes through the selects over the whole row.
template <bool CACHED, bool VEC, bool SMALL>
__global__ void __launch_bounds__(SAMPLE_THREADS, 2)
sample_kernel(int* __restrict__ out_ids, const float* __restrict__ logits, int vocab, int per_block, int values_bytes,
              const int* __restrict__ row_slot, const float* __restrict__ temperature,
              const int* __restrict__ top_k, const float* __restrict__ top_p,
              const float* __restrict__ penalty, const uint32_t* __restrict__ seen, int seen_words,
              const unsigned long long* __restrict__ rng_key, unsigned int* __restrict__ rng_counter, int team_size) {
  static_assert(!(CACHED && SMALL), "the small form keeps no values");
  __shared__ SampleShared sh;
  extern __shared__ __align__(16) unsigned char dynamic[];
  float* values = reinterpret_cast<float*>(dynamic);  // the slice; in the first block later the candidates' ids and values
  uint32_t* hist = reinterpret_cast<uint32_t*>(dynamic + values_bytes);

  pdl_trigger();
  team_arrive();
  pdl_wait(logits, row_slot, temperature, top_k, top_p, penalty, seen);
  Team team = {&sh, hist, team_size, (int)(blockIdx.x % team_size), 0};
  const int row = blockIdx.x / team_size, rank = team.rank;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int slot = row_slot[row];
  if (slot < 0) {  // the whole team
    team_wait();
    if (rank == 0 && threadIdx.x == 0) out_ids[row] = -1;
    return;
  }
  const int base = (int)min((long long)vocab, (long long)rank * per_block);
  const int n = min(per_block, vocab - base);
  RowView view;
  view.logits = logits + (size_t)row * vocab + base;
  view.penalty = penalty[row];
  view.seen = (seen != nullptr && view.penalty > 1.0f) ? seen + (size_t)slot * seen_words + base / 32 : nullptr;
  const float temp = temperature[row];
  const int k = top_k[row];
  const bool few = !SMALL && temp > 1e-5f && k > 0 && k < vocab;  // candidates are gathered first
  SmallShared* small = reinterpret_cast<SmallShared*>(dynamic);   // SMALL: where the others keep values

  // The one pass over the logits: penalty, and every thread's largest value (the first of equals).  For a small top_k a
  // histogram of the order keys' top 12 bits says where to cut: of the threads' largest values if they are at least twice
  // as many as k (there are then k elements at or above the cut, and hardly more), else of all values.
  const bool of_largest = k <= SAMPLE_THREADS / 2;
  if (few)
    for (int b = threadIdx.x; b < SAMPLE_FINE_BINS; b += SAMPLE_THREADS) hist[b] = 0u;
  if (few) __syncthreads();
  float best = -INFINITY; int best_i = -1;
  auto take = [&](int i, float a) {
    if (CACHED) values[i] = a;
    if (a > best) { best = a; best_i = i; }  // indices rise: the first maximum is kept
    if (few && !of_largest) atomicAdd(&hist[order_key(a) >> 20], 1u);
  };
  // every element of this thread, with the penalty; `ahead` loads in flight
  auto visit_by = [&](auto ahead, auto&& f) {
    if (VEC) {
      constexpr int UNROLL = decltype(ahead)::value;
      const int quads = n / 4;
      const float4* src = reinterpret_cast<const float4*>(view.logits);
      for (int q0 = threadIdx.x; q0 < quads; q0 += UNROLL * SAMPLE_THREADS) {
        float4 v[UNROLL]; uint32_t bits[UNROLL];
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
          const int q = q0 + u * SAMPLE_THREADS;
          v[u] = q < quads ? src[q] : make_float4(0.f, 0.f, 0.f, 0.f);
          bits[u] = (q < quads && view.seen != nullptr) ? view.seen[q >> 3] >> (4 * (q & 7)) : 0u;
        }
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
          const int q = q0 + u * SAMPLE_THREADS;
          if (q < quads) {
            float a[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              if ((bits[u] >> e) & 1u) a[e] = a[e] > 0.f ? a[e] / view.penalty : a[e] * view.penalty;
              f(4 * q + e, a[e]);
            }
          }
        }
      }
    } else {
      for (int i = threadIdx.x; i < n; i += SAMPLE_THREADS) f(i, view.adjusted(i));
    }
  };
  auto visit = [&](auto&& f) { visit_by(std::integral_constant<int, 4>(), f); };
  visit(take);
  auto adjusted = [&](int i) { return CACHED ? values[i] : view.adjusted(i); };
  auto each = [&](auto&& f) {  // (for the selects)
    if constexpr (CACHED) {
      for (int i = threadIdx.x; i < n; i += SAMPLE_THREADS) f(i, values[i]);
    } else {
      visit_by(std::integral_constant<int, 2>(), f);
    }
  };

  if (few && of_largest) atomicAdd(&hist[best_i < 0 ? 0 : order_key(best) >> 20], 1u);
  // (larger value, smaller place) as one number; 0 where nothing lies above minus infinity
  uint64_t packed = best_i < 0 ? 0ull : ((uint64_t)order_key(best + 0.0f) << 32) | (uint32_t)~(uint32_t)(base + best_i);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const uint64_t other = __shfl_xor_sync(0xffffffffu, (unsigned long long)packed, o);
    packed = other > packed ? other : packed;
  }
  if (lane == 0) sh.scan[warp] = packed;
  const uint32_t own_key = best_i < 0 ? 0u : order_key(best + 0.0f);  // (both zeros alike: which of them is first in `best` is chance)
  if (SMALL) {
    uint32_t group = own_key;
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) group = max(group, __shfl_xor_sync(0xffffffffu, group, o));
    if ((lane & 7) == 0) small->own_key[threadIdx.x >> 3] = group;
    if (threadIdx.x == 0) small->count = 0;
  }
  __syncthreads();
  if (threadIdx.x < SAMPLE_TEAM) {
    for (int w = 0; w < SAMPLE_WARPS; ++w) packed = sh.scan[w] > packed ? sh.scan[w] : packed;
  }
  __syncthreads();

  // This block's candidates, in index order.  Cut at its own k-th largest value (what the row keeps lies at or above the row's
  // k-th largest, which is no smaller) where all blocks together then keep few; at the row's, by the histograms of all blocks, for
  // a larger k: 500 of 128,256 at each of eight blocks' own leave more than there is room for, and the selects over the whole row
  // took 195 us for 64 rows (now 91).
  int* my_id = reinterpret_cast<int*>(hist);
  float* my_val = reinterpret_cast<float*>(hist) + SAMPLE_HIST_BYTES / 8;
  if (few) {
    uint32_t cut;
    if (of_largest || (long long)k * team_size <= SAMPLE_CANDIDATES / 4) {
      cut = find_cut<false>(hist, k, team);
    } else {
      team_wait();
      team_sync();  // every block's histogram is complete
      cut = find_cut<true>(hist, k, team);
      team_arrive();
    }
    const int count = gather(adjusted, [&](int i) { return base + i; }, n, cut, SAMPLE_HIST_BYTES / 8, &sh, my_id, my_val);
    if (threadIdx.x == 0) sh.count = count <= SAMPLE_HIST_BYTES / 8 ? count : -1;
  }

  team_wait();  // every block of the team runs: its shared memory may be written
  if (SMALL)
    for (int e = threadIdx.x; e < SAMPLE_GROUPS * team_size; e += SAMPLE_THREADS)
      of_block(small->group_key, e / SAMPLE_GROUPS)[rank * SAMPLE_GROUPS + e % SAMPLE_GROUPS] = small->own_key[e % SAMPLE_GROUPS];
  if ((int)threadIdx.x < team_size) {
    of_block(sh.best, threadIdx.x)[rank] = packed;
    if (rank == 0) {
      const unsigned int counter = rng_counter[slot];
      __syncwarp(__activemask());
      if (threadIdx.x == 0) rng_counter[slot] = counter + 1;
      *of_block(&sh.draw, threadIdx.x) =
          (unsigned int)(sm64(rng_key[slot] + ((uint64_t)counter + 1ull) * 0x9E3779B97F4A7C15ull) >> 32);
    }
  }
  team_sync();
  packed = 0;
  for (int r = 0; r < team_size; ++r) packed = sh.best[r] > packed ? sh.best[r] : packed;
  const uint32_t best_key = (uint32_t)(packed >> 32);
  const float row_max = packed == 0 ? -INFINITY
                                    : __uint_as_float((best_key & 0x80000000u) ? (best_key & 0x7fffffffu) : ~best_key);
  const int row_arg = packed == 0 ? 0 : (int)~(uint32_t)packed;
  if (temp <= 1e-5f || packed == 0) {  // (a row without a value above minus infinity has no probabilities: its first id)
    if (rank == 0 && threadIdx.x == 0) out_ids[row] = row_arg;
    return;
  }

  const float p = top_p[row];
  if (SMALL) {
    const int groups = SAMPLE_GROUPS * team_size;
    bool served = k > 0 && k < vocab && 2 * k <= groups;
    if (served) {
      if ((int)threadIdx.x < groups) {
        const uint32_t key = small->group_key[threadIdx.x];
        int above = 0, equal = 0;
#pragma unroll 4
        for (int j = 0; j < groups; j += 4) {
          const uint4 other = *reinterpret_cast<const uint4*>(&small->group_key[j]);
          above += (other.x > key) + (other.y > key) + (other.z > key) + (other.w > key);
          equal += (other.x == key) + (other.y == key) + (other.z == key) + (other.w == key);
        }
        if (above < k && k <= above + equal) small->cut = key;  // (all who write it write the same)
      }
      __syncthreads();
      const uint32_t cut = max(small->cut, SAMPLE_LOWEST_KEY + 1);  // fewer values than k groups: all that have a mass are kept
      SmallShared* first = of_block(small, 0);
      auto list = [&](uint32_t low) {  // of this block, what lies at or above `low`
        if (own_key < low) return;
        bool room = true;
        visit([&](int i, float a) {
          if (room && order_key(a + 0.0f) >= low) {
            const int place = atomicAdd(&first->count, 1);
            room = place < SAMPLE_CANDIDATES;
            if (room) {
              first->id[place] = base + i;
              first->value[place] = a;
            }
          }
        });
      };
      list(cut);
      team_sync();  // the candidates are there
      int count = first->count;
      served = count <= SAMPLE_THREADS;
      team_sync();  // everybody has read how many they are
      if (!served) {
        if (rank == 0 && threadIdx.x == 0) small->count = 0;
        team_sync();
        list(cut + 1);
        team_sync();
        count = first->count;
        if (count < k) {  // the rest are the first values equal to the cut (of zeros, those without a sign come first)
          served = send_ties([&](int i) { return order_key(adjusted(i)) == cut; }, adjusted, n, base, k - count, first, count,
                             sh.warp_count, small->ties, team);
          count = k;
        } else if (count <= SAMPLE_CANDIDATES) {  // the first block cuts once more, by the top 12 bits of the keys
          if (rank == 0 && count > SAMPLE_THREADS) {
            int* few_id = reinterpret_cast<int*>(hist);
            float* few_val = reinterpret_cast<float*>(hist) + SAMPLE_THREADS;
            for (int b = threadIdx.x; b < SAMPLE_FINE_BINS; b += SAMPLE_THREADS) hist[b] = 0u;
            __syncthreads();
            for (int i = threadIdx.x; i < count; i += SAMPLE_THREADS) atomicAdd(&hist[order_key(small->value[i]) >> 20], 1u);
            __syncthreads();
            const uint32_t fine = find_cut<false>(hist, k, team);
            const int left = gather([&](int i) { return small->value[i]; }, [&](int i) { return small->id[i]; }, count, fine,
                                    SAMPLE_THREADS, &sh, few_id, few_val);
            if (left <= SAMPLE_THREADS && (int)threadIdx.x < left) {
              small->id[threadIdx.x] = few_id[threadIdx.x];
              small->value[threadIdx.x] = few_val[threadIdx.x];
            }
            if (threadIdx.x == 0) small->count = left;
          }
          team_sync();
          count = first->count;
          served = count <= SAMPLE_THREADS;
        }
        team_sync();
      }
      if (served) {
        if (rank != 0) return;
        uint64_t* order = reinterpret_cast<uint64_t*>(hist);
        const int id = ranked_id(small->id, small->value, count, k, temp, p, row_max, row_arg, order, order + SAMPLE_THREADS, team);
        if (threadIdx.x == 0) out_ids[row] = id;
        return;
      }
    }
  }
  bool compact = few;
  int counts[SAMPLE_TEAM];
  int all = 0;
#pragma unroll
  for (int r = 0; r < SAMPLE_TEAM; ++r) {
    counts[r] = (few && r < team_size) ? *of_block(&sh.count, r) : 0;
    compact = compact && counts[r] >= 0;
    all += counts[r];
  }
  compact = compact && all <= SAMPLE_CANDIDATES;
  if (compact) {
    if (rank == 0) {
      int* ids = reinterpret_cast<int*>(values);
      float* vals = values + SAMPLE_CANDIDATES;
      int at = 0;
#pragma unroll
      for (int r = 0; r < SAMPLE_TEAM; ++r) {
        if (r < team_size) {
          const int* from_id = of_block(my_id, r);
          const float* from_val = of_block(my_val, r);
          for (int i = threadIdx.x; i < counts[r]; i += SAMPLE_THREADS) {
            ids[at + i] = from_id[i];
            vals[at + i] = from_val[i];
          }
        }
        at += counts[r];
      }
      team_sync();  // the candidates are here: the other blocks may leave
      if (all > SAMPLE_NARROW && k <= SAMPLE_THREADS / 2) {
        for (int b = threadIdx.x; b < SAMPLE_FINE_BINS; b += SAMPLE_THREADS) hist[b] = 0u;
        __syncthreads();
        for (int i = threadIdx.x; i < all; i += SAMPLE_THREADS) atomicAdd(&hist[order_key(vals[i]) >> 20], 1u);
        __syncthreads();
        int* few_id = reinterpret_cast<int*>(hist);
        float* few_val = reinterpret_cast<float*>(hist) + SAMPLE_THREADS;
        const uint32_t cut = find_cut<false>(hist, k, team);
        const int count = gather([&](int i) { return vals[i]; }, [&](int i) { return ids[i]; }, all, cut, SAMPLE_THREADS, &sh,
                                 few_id, few_val);
        if (count <= SAMPLE_THREADS) {
          ids = few_id;
          vals = few_val;
          all = count;
        }
      }
      long long place;
      if (all <= SAMPLE_THREADS) {
        uint64_t* order = reinterpret_cast<uint64_t*>(hist) + SAMPLE_THREADS;  // beyond the candidates that may lie there
        place = ranked_place(threadIdx.x < all ? vals[threadIdx.x] : 0.f, all, k, temp, p, row_max, order,
                             order + SAMPLE_THREADS, team);
      } else {
        auto value = [&](int i) { return vals[i]; };
        auto every = [&](auto&& f) { for (int i = threadIdx.x; i < all; i += SAMPLE_THREADS) f(i, vals[i]); };
        place = sample_place<false>(value, every, all, 0, all, k, temp, p, row_max, false, team);
      }
      if (threadIdx.x == 0) out_ids[row] = place >= 0 ? ids[place] : row_arg;
    } else {
      team_sync();
    }
    return;
  }
  team_sync();  // the counts are read; the histograms start anew
  const bool wide = n > 65535 * SAMPLE_HIST_COPIES;
  const long long place = sample_place<true>(adjusted, each, n, base, vocab, k, temp, p, row_max, wide, team);
  if (rank == 0 && threadIdx.x == 0) out_ids[row] = place >= 0 ? (int)place : row_arg;
  team_sync();  // nobody leaves while its sums may still be read
}

// Marks token ids as seen in their slot's bitmap (the history the repetition penalty looks at).
__global__ void mark_seen_kernel(uint32_t* __restrict__ seen, int seen_words, const int* __restrict__ slots,
                                 const int* __restrict__ ids, int n, int vocab) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int slot = slots[i], id = ids[i];
  if (slot < 0 || id < 0 || id >= vocab) return;
  atomicOr(&seen[(size_t)slot * seen_words + (id >> 5)], 1u << (id & 31));
}

}  // namespace xrt

namespace xrt {

// One limit for every launch of a form: setting a smaller one beside a launch of another thread would take it its room.
template <bool CACHED, bool VEC, bool SMALL>
static auto sample_form(cudaError_t& err) {
  err = allow_shared_memory_once<sample_kernel<CACHED, VEC, SMALL>>(SAMPLE_CACHED_BYTES + SAMPLE_HIST_BYTES);
  return sample_kernel<CACHED, VEC, SMALL>;
}

}  // namespace xrt

// logits: [n_rows, vocab] 32-bit.  Per row: its slot (< 0 = padding, id -1), temperature, top_k
// (0 = all), top_p (>= 1 = all), repetition penalty (<= 1 = none).  seen: [slots, seen_words]
// bitmaps or null.  rng_key / rng_counter: per slot.  largest_top_k: where the caller knows that every row is greedy or has a
// top_k of at least 1, the largest of those, else 0; it chooses the form of the kernel and changes no result.
XRT_EXPORT int xrt_sample(int* out_ids, const float* logits, int n_rows, int vocab, const int* row_slot,
                          const float* temperature, const int* top_k, const float* top_p, const float* penalty,
                          const unsigned int* seen, int seen_words, const unsigned long long* rng_key,
                          unsigned int* rng_counter, int largest_top_k, cudaStream_t stream) {
  if (n_rows < 0 || vocab <= 0) return XRT_ERR_ARGUMENT;
  if (seen != nullptr && seen_words * 32 < vocab) return XRT_ERR_ARGUMENT;
  if (n_rows == 0) return XRT_OK;
  const int sms = xrt::multiprocessors();
  // blocks of a team: as many as it takes to bring a slice to 4,096 logits (smaller ones are read in less time than a team takes
  // to meet), or, where the rows alone occupy the multiprocessors, as keep it at 4,096 (256 rows of 5,000 logits, one block against
  // two: 20.7 against 26.6 us); half as many while the rows alone bring more than four blocks a multiprocessor
  int team = 1;
  while (team < xrt::SAMPLE_TEAM && (long long)team * (n_rows >= sms ? 2 * 4096 - 1 : 4096) < vocab) team *= 2;
  while (team > 2 && (long long)team * n_rows > 4ll * sms) team /= 2;
  // The SMALL form where those blocks would take more than one round (two run on a multiprocessor at a time): a team of no more than
  // four, as run all at once, with at least twice as many groups of lanes as the largest top_k.
  int small_team = team < 4 ? team : 4;
  while (small_team > 2 && (long long)small_team * n_rows > 2ll * sms) small_team /= 2;
  const bool small = (long long)team * n_rows > 2ll * sms && largest_top_k > 0 && largest_top_k < vocab && small_team > 1 &&
                     2 * largest_top_k <= small_team * xrt::SAMPLE_GROUPS;
  if (small) team = small_team;
  const long long per = ((long long)vocab + team * 32 - 1) / (team * 32) * 32;
  const bool cached = !small && per * 4 <= xrt::SAMPLE_CACHED_BYTES;
  const bool vec = vocab % 4 == 0 && ((uintptr_t)logits & 15) == 0;
  int values_bytes = cached ? (int)per * 4 : 0;
  if (small) values_bytes = (int)((sizeof(xrt::SmallShared) + 15) / 16 * 16);
  else if (values_bytes < xrt::SAMPLE_CANDIDATES * 8) values_bytes = xrt::SAMPLE_CANDIDATES * 8;
  const size_t smem = (size_t)values_bytes + xrt::SAMPLE_HIST_BYTES;
  cudaError_t err = cudaSuccess;
  auto kernel = small ? (vec ? xrt::sample_form<false, true, true>(err) : xrt::sample_form<false, false, true>(err))
                : cached ? (vec ? xrt::sample_form<true, true, false>(err) : xrt::sample_form<true, false, false>(err))
                         : (vec ? xrt::sample_form<false, true, false>(err) : xrt::sample_form<false, false, false>(err));
  if (err != cudaSuccess) return (int)err;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3((unsigned)n_rows * team);
  config.blockDim = dim3(xrt::SAMPLE_THREADS);
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  cudaLaunchAttribute attrs[2];
  attrs[0].id = cudaLaunchAttributeClusterDimension;
  attrs[0].val.clusterDim.x = team; attrs[0].val.clusterDim.y = 1; attrs[0].val.clusterDim.z = 1;
  attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attrs[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attrs;
  config.numAttrs = xrt::pdl_enabled() ? 2 : 1;
  cudaLaunchKernelEx(&config, kernel, out_ids, logits, vocab, (int)per, values_bytes, row_slot, temperature, top_k, top_p,
                     penalty, (const uint32_t*)seen, seen_words, rng_key, rng_counter, team);
  return xrt::launch_status();
}

XRT_EXPORT int xrt_mark_seen(unsigned int* seen, int seen_words, const int* slots, const int* ids, int n,
                             int vocab, cudaStream_t stream) {
  if (n < 0 || vocab <= 0 || seen_words * 32 < vocab) return XRT_ERR_ARGUMENT;
  if (n == 0) return XRT_OK;
  xrt::mark_seen_kernel<<<(n + 255) / 256, 256, 0, stream>>>(seen, seen_words, slots, ids, n, vocab);
  return xrt::launch_status();
}
