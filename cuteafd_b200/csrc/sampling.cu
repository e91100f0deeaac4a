// Exact full-vocabulary target sampling on the GPU, a cluster of thread blocks per logit row, plus the
// accept-prefix scan of sample-match speculative verification.
//
// Filter order: allowed-token mask -> temperature -> min_p -> top_k (exactly k, lowest id wins a
// boundary tie) -> top_p (smallest descending prefix reaching the mass) -> draw.  The uniform is a
// pure function of (seed, absolute position) (SplitMix64), so row layout cannot change a token.
//
// Every filter is "the smallest prefix of the order (descending value, ascending id) whose
// cumulative count / probability mass reaches a target".  Probability mass is a 2^-44 fixed-point
// integer, so sums are associative and the result does not depend on thread timing: the same row
// always yields the same token.
//
// One cluster of one to eight blocks per row, each with its share of the vocabulary in shared memory as
// order-preserving 32-bit keys.  What bounds the kernel is the number of dependent passes, not the
// 0.6 MB a row is read once: with one block per row, walking the row from L2 in every pass, eight
// rows of 151936 took 371 us and 32 rows of 129280 666 us, then 27 and 35 us, with the quick pass 18
// (top-k 50) and 33 (top-p 0.9).  One histogram over
// (maximum - value) in steps of 1/8 says how far down the first filter can reach; the tokens above
// that line, a few hundred for the settings that chats use, are gathered into one block, sorted,
// and all filters and the draw are prefix sums over the sorted list.  The shared atomics of that
// histogram, up to four to a token, were the longest part: where the threads' best tokens can say
// beforehand which tokens may matter (the quick pass), the others meet none.  When more than 2048
// tokens are above the line the selections are four-level radix descents over the keys in the cluster.
//
// Reference counterparts: native/shared/cuda/sampling_gpu.cu (row parameters and status codes
// sampling_gpu.h:82-120), semantics in rust/crates/cuteafd-core/src/target_sampling.rs:9-215.
#include "cafd_api.h"
#include "common.cuh"
#include <cooperative_groups.h>

namespace cafd {
namespace cg = cooperative_groups;

constexpr int kSampleThreads = 512;              // at 64 registers a thread two blocks share an SM: 32 rows are one wave (1024 threads: two waves, 67 us)
constexpr int kSampleBins = 256;
constexpr int kSampleList = 2048;                // tokens that the sorted list holds
constexpr int kSampleNear = 1024;                // threads' best tokens above the quick pass's line
// Tokens of a block's slice from which the quick pass gains more than its barriers cost: with top-k, and without.  Without it / with it, us: 8 rows of
// 32000 (slices of 4000), top-k 50, 14.7 / 14.9, top-p 0.9 14.6 / 17.1; 4 of 50000 16.6 / 15.2 and 16.3 / 18.3; 20 of 100000 30 / 24 and 30.5 / 27.7; 8 of
// 151936 27.7 / 18.2 and 28.0 / 23.9, flat rows of them 29.7 / 20.0 and 103 / 97.5.  Without top-k a row's threads must be more than a list holds to
// show that it is flat: eight blocks (256 flat rows of 32000 on two blocks each 251 / 302).
constexpr int kSampleQuickK = 6 * 1024, kSampleQuick = 12 * 1024;
constexpr int kSampleNearList = 1024;            // tokens above it that a block notes
constexpr int kSampleSmemKeys = 48 * 1024;       // keys of a slice kept in shared memory; longer slices are read again in every pass
constexpr int kSampleKeysPair = 20 * 1024;       // up to this many two blocks share an SM
constexpr int kLimbKeys = 1 << 17;               // slice length up to which 15-bit limbs of the masses add up in 32 bits
constexpr float kGreedyEps = 1.0e-5f;

struct SampleRow {          // 64 bytes
  float temperature, top_p, min_p;
  int top_k;                // <= 0: no limit
  unsigned long long seed;
  long long position;
  long long mask_word0;     // first 32-bit word of this row's allowed-token bitmask in `masks`, < 0: none
  int logits_row;           // row of the logits matrix
  int pad[5];
};

enum : int { kSampleOk = 0, kSampleNonFinite = 1, kSampleEmptyMask = 2, kSampleBadParam = 3 };

__device__ __forceinline__ uint32_t order_key(float x) {
  const uint32_t b = __float_as_uint(x + 0.0f);          // both zeros are one value
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

__device__ __forceinline__ float splitmix_uniform(unsigned long long seed, long long position) {
  unsigned long long x = seed + 0x7F4A7C159E3779B9ull + static_cast<unsigned long long>(position) * 0x9E3779B97F4A7C15ull +
                         0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  x ^= x >> 31;
  return static_cast<float>(x >> 40) * (1.0f / 16777216.0f);
}

struct Cut { uint32_t key; int id; };     // members: key > cut.key, or key == cut.key and id <= cut.id

// Histogram of one pass: a count and a mass per bin.  Masses are below 2^45: three 15-bit limbs, each with native 32-bit shared
// atomics (a 64-bit shared add is a compare-and-swap loop); a slice too long for their sums takes two whole words.
struct SampleHist {
  unsigned int cnt[kSampleBins];
  unsigned int limb[3][kSampleBins];
};

struct SampleShared {
  SampleHist hist[2];
  unsigned long long list[kSampleList];       // key << 32 | ~id: descending = the order
  int near_id[kSampleNearList];               // places of the slice's tokens above the quick pass's line
  unsigned long long near_mass[kSampleThreads / 32], row_mass;      // this block's share of the row's mass
  int n_near, near_bin, near_flat;
  unsigned long long scan[32];
  int counts[32];
  float red_v[32];
  int red_i[32], red_c[32], red_bad[32];
  float row_v;
  int row_i, row_c, row_bad;                  // this block's share of the row's maximum, argmax, allowed tokens, non-finite logits
  int n_list, ties, pick_id, bin;
  unsigned long long tie_mass, acc_m, level_acc[2], level_total;      // of a descent: sum above the level's bin, and the whole
  int level_bin[2];
  unsigned int acc_c;
};

__device__ __forceinline__ float key_value(uint32_t key) {
  return __uint_as_float((key & 0x80000000u) ? (key ^ 0x80000000u) : ~key);
}

// Probability mass relative to the best token as a 2^-44 fixed-point integer (exp on the special-function unit: the same input
// always gives the same bits, which is all the selections need).
__device__ __forceinline__ unsigned long long mass_of(float xp, float maxp) {
  return __float2ull_rn(fast_exp2((xp - maxp) * 1.4426950408889634f) * 17592186044416.0f);
}

// Inclusive sums over the block's threads in thread order.
template <typename T>
__device__ __forceinline__ T block_scan(T v, T* warp_tot) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T w = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += w;
  }
  __syncthreads();
  if (lane == 31) warp_tot[wid] = v;
  __syncthreads();
  T before = 0;
#pragma unroll
  for (int w = 0; w < kSampleThreads / 32; ++w) before += w < wid ? warp_tot[w] : T(0);
  return v + before;
}

__device__ __forceinline__ unsigned long long mass_target(double frac, bool strict, unsigned long long total) {
  const double t = frac * static_cast<double>(total);
  unsigned long long ti = strict ? static_cast<unsigned long long>(floor(t)) + 1ull : static_cast<unsigned long long>(ceil(t));
  if (ti > total) ti = total;
  return ti < 1ull ? 1ull : ti;
}

// One block's slice of a row: keys in shared memory, or the logits themselves when the slice is too long for it.  Key 0 (no finite
// value has it) stands for a token that is masked out or below min_p.
struct SampleSlice {
  uint32_t* keys;          // shared memory, or null
  const float* x;
  const uint32_t* mask;
  int id0, n;
  float temp, thresh, maxp;
  bool use_minp;
  __device__ __forceinline__ uint32_t make(int j) const {
    const int i = id0 + j;
    if (mask && !((mask[i >> 5] >> (i & 31)) & 1u)) return 0u;
    const float xp = x[i] / temp;
    return use_minp && !(xp >= thresh) ? 0u : order_key(xp);
  }
  __device__ __forceinline__ uint32_t key(int j) const { return keys ? keys[j] : make(j); }
  // steps of 1/8 below the maximum: never falls as the value does, so the bins are stretches of the order
  __device__ __forceinline__ int bin(float xp) const { return min(kSampleBins - 1, max(0, static_cast<int>((maxp - xp) * 8.0f))); }
};

__device__ __forceinline__ void hist_clear(SampleHist& h) {
  for (int i = threadIdx.x; i < kSampleBins; i += kSampleThreads) {
    h.cnt[i] = 0;
    h.limb[0][i] = 0; h.limb[1][i] = 0; h.limb[2][i] = 0;
  }
}
__device__ __forceinline__ void hist_add_mass(SampleHist& h, int b, unsigned long long m, bool wide) {
  if (wide) {                                    // two words, the carry of the lower from the value it had
    const unsigned int lo = static_cast<unsigned int>(m), was = atomicAdd(&h.limb[0][b], lo);
    const unsigned int hi = static_cast<unsigned int>(m >> 32) + (was + lo < was ? 1u : 0u);
    if (hi) atomicAdd(&h.limb[1][b], hi);
    return;
  }
  const unsigned int l0 = static_cast<unsigned int>(m) & 0x7fffu, l1 = static_cast<unsigned int>(m >> 15) & 0x7fffu, l2 = static_cast<unsigned int>(m >> 30);
  if (l0) atomicAdd(&h.limb[0][b], l0);
  if (l1) atomicAdd(&h.limb[1][b], l1);
  if (l2) atomicAdd(&h.limb[2][b], l2);
}
// Thread t < 256 gets bin b's count and mass over the whole cluster (after the cluster's barrier).
template <int kC>
__device__ __forceinline__ void hist_total(cg::cluster_group& cluster, SampleHist& h, int b, bool wide, unsigned int& c, unsigned long long& m) {
  c = 0; m = 0;
#pragma unroll
  for (int r = 0; r < kC; ++r) {
    const SampleHist* o = cluster.map_shared_rank(&h, r);
    c += o->cnt[b];
    if (wide) m += o->limb[0][b] + (static_cast<unsigned long long>(o->limb[1][b]) << 32);
    else m += o->limb[0][b] + (static_cast<unsigned long long>(o->limb[1][b]) << 15) + (static_cast<unsigned long long>(o->limb[2][b]) << 30);
  }
}

// Smallest prefix of the order, inside `cut`, whose cumulative metric reaches `target_frac` (by_mass: a fraction of the cut's total
// mass, strict = "exceeds"; else a count).  Returns the new cut; its id is the last member of the prefix.  All threads of the cluster
// call this with identical arguments.
template <int kC>
__device__ Cut select_prefix(cg::cluster_group& cluster, const SampleSlice& s, Cut cut, bool by_mass, double frac, bool strict,
                             long long count_target, bool wide, SampleShared& sh) {
  const int tid = threadIdx.x, rank = static_cast<int>(cluster.block_rank());
  unsigned long long target = 0, acc = 0;
  uint32_t prefix = 0;
  for (int level = 0; level < 4; ++level) {
    const int shift = 24 - 8 * level;
    SampleHist& h = sh.hist[level & 1];      // last read two levels ago, before the barrier of the level between
    hist_clear(h);
    if (tid == 0) { sh.level_bin[level & 1] = 0; sh.level_acc[level & 1] = acc; }
    __syncthreads();
    for (int j = tid; j < s.n; j += kSampleThreads) {
      const uint32_t key = s.key(j);
      if (!key || key < cut.key || (key == cut.key && s.id0 + j > cut.id)) continue;
      if (level > 0 && (key >> (shift + 8)) != prefix) continue;
      const int b = (key >> shift) & 255u;
      if (by_mass) hist_add_mass(h, b, mass_of(key_value(key), s.maxp), wide);
      else atomicAdd(&h.cnt[b], 1u);
    }
    cluster.sync();
    unsigned int c = 0;
    unsigned long long m = 0;
    const int b = 255 - tid;                 // thread order = descending keys
    if (tid < kSampleBins) hist_total<kC>(cluster, h, b, wide, c, m);
    const unsigned long long v = by_mass ? m : c;
    const unsigned long long incl = block_scan(v, sh.scan);
    if (level == 0) {
      if (tid == kSampleThreads - 1) sh.level_total = incl;
      __syncthreads();
      const unsigned long long total = sh.level_total;
      if (by_mass) target = mass_target(frac, strict, total);
      else target = min(max(1ull, static_cast<unsigned long long>(count_target)), max(1ull, total));
    }
    if (tid < kSampleBins && v > 0 && acc + incl >= target && acc + incl - v < target) { sh.level_bin[level & 1] = b; sh.level_acc[level & 1] = acc + incl - v; }
    __syncthreads();
    acc = sh.level_acc[level & 1];
    prefix = (prefix << 8) | static_cast<uint32_t>(sh.level_bin[level & 1]);
  }
  // ties of the pivot value: how many are needed, then the id of that tie (ascending ids: blocks in rank order, a thread a run of ids)
  const int chunk = (s.n + kSampleThreads - 1) / kSampleThreads;
  const int lo = min(s.n, tid * chunk), hi = min(s.n, lo + chunk);
  int mine = 0;
  for (int j = lo; j < hi; ++j) {
    const uint32_t key = s.key(j);
    if (key == prefix && key && (key > cut.key || s.id0 + j <= cut.id)) ++mine;
  }
  const int incl = block_scan(mine, sh.counts);
  if (tid == kSampleThreads - 1) sh.ties = incl;
  if (tid == 0) sh.pick_id = -1;
  cluster.sync();
  int before = 0, n_ties = 0;
#pragma unroll
  for (int r = 0; r < kC; ++r) {
    const int t = *cluster.map_shared_rank(&sh.ties, r);
    if (r < rank) before += t;
    n_ties += t;
  }
  const unsigned long long rest = target > acc ? target - acc : 1ull;
  const unsigned long long tie_mass = prefix ? mass_of(key_value(prefix), s.maxp) : 0ull;
  long long need = by_mass ? (tie_mass > 0 ? static_cast<long long>((rest + tie_mass - 1) / tie_mass) : 1) : static_cast<long long>(rest);
  need = min(max(need, 1ll), static_cast<long long>(n_ties));
  int seen = before + incl - mine;
  if (mine > 0 && seen < need && need <= seen + mine) {
    for (int j = lo; j < hi; ++j) {
      const uint32_t key = s.key(j);
      if (key == prefix && (key > cut.key || s.id0 + j <= cut.id) && ++seen == need) {
        for (int r = 0; r < kC; ++r) *cluster.map_shared_rank(&sh.pick_id, r) = s.id0 + j;
        break;
      }
    }
  }
  cluster.sync();        // (what another block reads of this call is read: a next call writes it behind barriers of its own)
  return Cut{prefix, sh.pick_id};
}

// All filters and the draw on the L tokens of sh.list (unsorted), of which the first nk in order are candidates; all_m: the row's mass.  One block.
__device__ int pick_from_list(SampleShared& sh, int L, int nk, bool use_k, bool use_p, unsigned long long all_m, float top_p, double u, float maxp,
                              int best_id) {
  const int tid = threadIdx.x;
  int pow2 = 2;
  while (pow2 < L) pow2 <<= 1;
  for (int j = L + tid; j < pow2; j += kSampleThreads) sh.list[j] = 0ull;
  __syncthreads();
  for (int k = 2; k <= pow2; k <<= 1)        // bitonic, descending
    for (int d = k >> 1; d > 0; d >>= 1) {
      for (int t = tid; t < pow2 / 2; t += kSampleThreads) {
        const int i = 2 * t - (t & (d - 1)), o = i + d;
        const unsigned long long a = sh.list[i], b = sh.list[o];
        if ((a < b) == ((i & k) == 0)) { sh.list[i] = b; sh.list[o] = a; }
      }
      __syncthreads();
    }
  constexpr int kPer = kSampleList / kSampleThreads;
  unsigned long long c[kPer];                // masses, then cumulative masses, at this thread's places of the list
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    const int i = kPer * tid + q;
    c[q] = i < nk ? mass_of(key_value(static_cast<uint32_t>(sh.list[i] >> 32)), maxp) : 0ull;
    if (q) c[q] += c[q - 1];
  }
  const unsigned long long own = c[kPer - 1], incl = block_scan(own, sh.scan);
#pragma unroll
  for (int q = 0; q < kPer; ++q) c[q] += incl - own;
  const unsigned long long before = incl - own;
  if (tid == kSampleThreads - 1) sh.acc_m = use_k ? incl : all_m;
  __syncthreads();
  unsigned long long total = sh.acc_m;
  if (use_p) {
    const unsigned long long t = mass_target(static_cast<double>(top_p), false, total);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kPer; ++q)
      if (c[q] >= t && (q ? c[q - 1] : before) < t) sh.acc_m = c[q];
    __syncthreads();
    total = sh.acc_m;
  }
  const unsigned long long t = mass_target(u, true, total);
  if (tid == 0) sh.pick_id = best_id;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kPer; ++q)
    if (c[q] >= t && (q ? c[q - 1] : before) < t) sh.pick_id = static_cast<int>(0xffffffffu - static_cast<uint32_t>(sh.list[kPer * tid + q]));
  __syncthreads();
  return sh.pick_id;
}

template <int kC>
__global__ void __launch_bounds__(kSampleThreads) sample_rows_kernel(const float* __restrict__ logits, int ld, int V, int slice,
                                                                     const SampleRow* __restrict__ rows,
                                                                     const uint32_t* __restrict__ masks,
                                                                     int* __restrict__ out_token, int* __restrict__ out_status) {
  pdl_wait();
  pdl_trigger();
  __shared__ SampleShared sh;
  extern __shared__ __align__(16) uint32_t sm_keys[];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = static_cast<int>(cluster.block_rank());
  const int out_row = blockIdx.x / kC;
  const SampleRow rp = rows[out_row];
  const float* x = logits + static_cast<size_t>(rp.logits_row) * ld;
  const uint32_t* mask = rp.mask_word0 >= 0 ? masks + rp.mask_word0 : nullptr;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int id0 = min(V, rank * slice), n = min(V - id0, slice);
  const bool in_smem = slice <= kSampleSmemKeys, wide = slice > kLimbKeys;

  const bool bad_param = !(rp.temperature >= 0.f && rp.temperature <= 2.0f) || !(rp.top_p > 0.f && rp.top_p <= 1.0f) ||
                         !(rp.min_p >= 0.f && rp.min_p <= 1.0f) || V <= 0;
  // ---- pass A: validation, max, lowest-id argmax; the logits stay in shared memory ---------------------
  float best = -INFINITY; int bi = 0x7fffffff; int cnt = 0, bad = 0;
  const bool greedy = rp.temperature < kGreedyEps || rp.top_k == 1, keep = in_smem && !greedy;
  const bool use_k = rp.top_k > 0 && rp.top_k < V, use_p = rp.top_p < 1.0f;
  const bool quick_pass = keep && (use_k ? slice >= kSampleQuickK : kC == 8 && slice >= kSampleQuick);
  auto take = [&](int i, float v, bool allowed) {
    const bool finite = isfinite(v);
    cnt += allowed;
    bad |= allowed && !finite;
    if (allowed && finite && (v > best || (v == best && i < bi))) { best = v; bi = i; }
  };
  int from = 0;
  if ((reinterpret_cast<uintptr_t>(x + id0) & 15u) == 0) {
    // Sixteen logits in flight per thread, four to a load: a slice starts at a multiple of four tokens, so four share a mask word.  Where
    // a slice leaves an SM one block, its loads in flight are the pass's rate: 256 greedy rows of 262144 tokens 209 us with eight 4-byte
    // loads, 148 with these, of 151936 90 and 76 (one block per row and four blocks per SM: 145 and 90).  Eight vector loads: 142 and 134,
    // their registers cost the second block where there is one.
    constexpr int kAhead = 4;
    const int n4 = n / 4;
    const uint4* x4 = reinterpret_cast<const uint4*>(x + id0);
    for (int c0 = tid; c0 < n4; c0 += kAhead * kSampleThreads) {
      uint4 v[kAhead];
      uint32_t in[kAhead];
#pragma unroll
      for (int q = 0; q < kAhead; ++q) {
        const int c = c0 + q * kSampleThreads;
        in[q] = c < n4 ? 0xfu : 0u;
        v[q] = c < n4 ? __ldcg(x4 + c) : uint4{0u, 0u, 0u, 0u};
      }
      if (mask) {
#pragma unroll
        for (int q = 0; q < kAhead; ++q) {
          const int i = id0 + 4 * (c0 + q * kSampleThreads);
          if (in[q]) in[q] = (__ldcg(mask + (i >> 5)) >> (i & 31)) & 0xfu;
        }
      }
#pragma unroll
      for (int q = 0; q < kAhead; ++q) {
        const int c = c0 + q * kSampleThreads, i = id0 + 4 * c;
        if (keep && c < n4) reinterpret_cast<uint4*>(sm_keys)[c] = v[q];
        take(i, __uint_as_float(v[q].x), in[q] & 1u);
        take(i + 1, __uint_as_float(v[q].y), (in[q] >> 1) & 1u);
        take(i + 2, __uint_as_float(v[q].z), (in[q] >> 2) & 1u);
        take(i + 3, __uint_as_float(v[q].w), (in[q] >> 3) & 1u);
      }
    }
    from = 4 * n4;
  }
  constexpr int kAhead = 8;                       // rows of another alignment, and a row's last tokens
  for (int j0 = from + tid; j0 < n; j0 += kAhead * kSampleThreads) {
    float v[kAhead];
    bool in[kAhead];
#pragma unroll
    for (int q = 0; q < kAhead; ++q) {
      const int j = j0 + q * kSampleThreads;
      in[q] = j < n;
      v[q] = in[q] ? __ldcg(x + id0 + j) : 0.f;
    }
    if (mask) {
#pragma unroll
      for (int q = 0; q < kAhead; ++q) {
        const int i = id0 + j0 + q * kSampleThreads;
        if (in[q]) in[q] = (__ldcg(mask + (i >> 5)) >> (i & 31)) & 1u;
      }
    }
#pragma unroll
    for (int q = 0; q < kAhead; ++q) {
      const int j = j0 + q * kSampleThreads;
      if (keep && j < n) sm_keys[j] = __float_as_uint(v[q]);
      take(id0 + j, v[q], in[q]);
    }
  }
  const float mine = best;                      // this thread's best token
  for (int o = 16; o; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    bad |= __shfl_xor_sync(0xffffffffu, bad, o);
  }
  if (lane == 0) { sh.red_v[wid] = best; sh.red_i[wid] = bi; sh.red_c[wid] = cnt; sh.red_bad[wid] = bad; }
  hist_clear(sh.hist[0]);
  if (quick_pass) hist_clear(sh.hist[1]);
  if (tid == 0) { sh.n_list = 0; sh.n_near = 0; sh.bin = kSampleBins - 1; }
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < kSampleThreads / 32; ++w) {
      const float ov = sh.red_v[w]; const int oi = sh.red_i[w];
      if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
      cnt += sh.red_c[w]; bad |= sh.red_bad[w];
    }
    sh.row_v = best; sh.row_i = bi; sh.row_c = cnt; sh.row_bad = bad;
  }
  cluster.sync();
  best = -INFINITY; bi = 0x7fffffff; cnt = 0; bad = 0;
#pragma unroll
  for (int r = 0; r < kC; ++r) {
    const SampleShared* o = cluster.map_shared_rank(&sh, r);
    const float ov = o->row_v; const int oi = o->row_i;
    if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    cnt += o->row_c; bad |= o->row_bad;
  }
  int status = kSampleOk;
  if (bad_param) status = kSampleBadParam;
  else if (cnt == 0) status = kSampleEmptyMask;
  else if (bad) status = kSampleNonFinite;
  if (status != kSampleOk || greedy) {          // the same for all blocks of the row
    if (rank == 0 && tid == 0) { out_token[out_row] = status != kSampleOk ? -1 : bi; out_status[out_row] = status; }
    cluster.sync();                             // no block leaves while another reads its share
    return;
  }
  // ---- candidates: allowed, scaled by temperature, min_p; counts and masses by distance from the maximum ---
  SampleSlice s;
  s.keys = nullptr; s.x = x; s.mask = mask; s.id0 = id0; s.n = n; s.temp = rp.temperature;
  s.maxp = best / rp.temperature;
  s.use_minp = rp.min_p > 0.f;
  s.thresh = s.use_minp ? s.maxp + static_cast<float>(log(static_cast<double>(rp.min_p))) : -INFINITY;
  float uf = splitmix_uniform(rp.seed, rp.position);
  uf = fminf(fmaxf(uf, 0.f), 0.99999994f);
  const double u = static_cast<double>(uf);
  int token = bi;
  bool flat = false;
  if (quick_pass) {
    // ---- quick pass.  The best tokens of the row's threads, some 4096, give a line: above it are top-k tokens at least or, without top-k, most
    // of those tokens' mass.  Only tokens above it meet a histogram and are noted; of the others what counts, without top-k, is their mass,
    // which needs no atomics.  Where the first filter reaches no further than the line, the noted tokens are all there is to sort; a row too
    // flat for that is left to the passes over all tokens.
    const bool masses = !use_k;
    if (mine > -INFINITY) {
      const float xp = key_value(order_key(mine / s.temp));
      if (!s.use_minp || xp >= s.thresh) {
        const int b = s.bin(xp);
        atomicAdd(&sh.hist[1].cnt[b], 1u);
        if (masses) hist_add_mass(sh.hist[1], b, mass_of(xp, s.maxp), wide);
      }
    }
    cluster.sync();
    unsigned int bc = 0;
    unsigned long long bm = 0;
    if (tid < kSampleBins) hist_total<kC>(cluster, sh.hist[1], tid, wide, bc, bm);
    const unsigned int tc = block_scan(bc, reinterpret_cast<unsigned int*>(sh.counts));
    const unsigned long long tm = masses ? block_scan(bm, sh.scan) : 0ull;
    if (tid == 0) { sh.near_bin = -1; sh.near_flat = 0; }
    if (tid == kSampleThreads - 1) { sh.acc_m = tm; sh.acc_c = tc; }
    __syncthreads();
    if (tid < kSampleBins && bc > 0) {
      if (masses) {
        // the threads' tokens hold most of the mass where it is concentrated: a line at a quarter of what may be left below, of theirs
        const double goal = use_p ? static_cast<double>(rp.top_p) : u, all = static_cast<double>(sh.acc_m), want = (0.75 + 0.25 * goal) * all;
        if (tc <= kSampleNear && static_cast<double>(tm) >= want && static_cast<double>(tm - bm) < want) sh.near_bin = tid;
        // more of them than a list holds reach the goal: so do more tokens, and nothing is asked about lists
        if (tc > kSampleList && static_cast<double>(tm) >= goal * all && static_cast<double>(tm - bm) < goal * all) sh.near_flat = 1;
      } else if (tc <= kSampleNear) {
        const unsigned int k = static_cast<unsigned int>(rp.top_k);
        if (tc >= k && tc - bc < k) sh.near_bin = tid;
        else if (tc < k && tc == sh.acc_c) sh.near_bin = kSampleBins - 1;       // few threads have any candidate: all of them
      }
    }
    __syncthreads();
    flat = sh.near_flat != 0;
    const int near = sh.near_bin;
    const bool try_near = near >= 0;
    if (try_near) {
      unsigned long long mass = 0;
      // below this no token is in the bins down to the line, or passes min_p (x / temperature, the bin and the threshold round once each)
      const float slack = 0.1f * s.temp + 1e-6f * fabsf(best);
      const float least = s.use_minp ? s.thresh * s.temp - 1e-6f * fabsf(s.thresh * s.temp) - slack : -INFINITY;
      const float cut = fmaxf(least, near < kSampleBins - 1 ? best - static_cast<float>(near + 1) * 0.125f * s.temp - slack : -INFINITY);
      auto visit = [&](int j, float xv, bool in) {
        if (!in || xv < (masses ? least : cut)) return;
        const float xp = s.temp == 1.0f ? xv : xv / s.temp;
        if (s.use_minp && !(xp >= s.thresh)) return;
        if (masses) mass += mass_of(xp, s.maxp);
        if (xv < cut) return;
        const float value = key_value(order_key(xp));      // one zero
        const int b = s.bin(value);
        if (b > near) return;
        atomicAdd(&sh.hist[0].cnt[b], 1u);
        if (masses) hist_add_mass(sh.hist[0], b, mass_of(value, s.maxp), wide);
        const int at = atomicAdd(&sh.n_near, 1);
        if (at < kSampleNearList) sh.near_id[at] = j;
      };
      for (int c = tid; c < (n + 3) / 4; c += kSampleThreads) {
        const uint4 v = reinterpret_cast<const uint4*>(sm_keys)[c];
        const int i = id0 + 4 * c;
        uint32_t in = 0xfu;
        if (mask) {
          in = 0;
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (4 * c + e < n) in |= ((mask[(i + e) >> 5] >> ((i + e) & 31)) & 1u) << e;
        }
        visit(4 * c, __uint_as_float(v.x), in & 1u);
        visit(4 * c + 1, __uint_as_float(v.y), (in & 2u) && 4 * c + 1 < n);
        visit(4 * c + 2, __uint_as_float(v.z), (in & 4u) && 4 * c + 2 < n);
        visit(4 * c + 3, __uint_as_float(v.w), (in & 8u) && 4 * c + 3 < n);
      }
      if (masses)
        for (int o = 16; o; o >>= 1) mass += __shfl_xor_sync(0xffffffffu, mass, o);
      if (lane == 0) sh.near_mass[wid] = mass;
      __syncthreads();
      if (tid == 0) {
        for (int w = 1; w < kSampleThreads / 32; ++w) mass += sh.near_mass[w];
        sh.row_mass = mass;
      }
      cluster.sync();
      unsigned long long all_m = 0;
      bool quick = true;
#pragma unroll
      for (int r = 0; r < kC; ++r) {
        const SampleShared* o = cluster.map_shared_rank(&sh, r);
        all_m += o->row_mass;
        quick &= o->n_near <= kSampleNearList;
      }
      bc = 0; bm = 0;
      if (tid < kSampleBins) hist_total<kC>(cluster, sh.hist[0], tid, wide, bc, bm);
      const unsigned int cc = block_scan(bc, reinterpret_cast<unsigned int*>(sh.counts));
      const unsigned long long cm = masses ? block_scan(bm, sh.scan) : 0ull;
      if (tid == kSampleThreads - 1) { sh.bin = -1; sh.acc_c = cc; }
      __syncthreads();
      // (with top-k, fewer than k tokens down to the line are all candidates)
      const unsigned long long first = use_k ? min(static_cast<unsigned long long>(rp.top_k), static_cast<unsigned long long>(sh.acc_c))
                                             : mass_target(use_p ? static_cast<double>(rp.top_p) : u, !use_p, all_m);
      __syncthreads();
      if (tid < kSampleBins) {
        const unsigned long long at = use_k ? cc : cm, own = use_k ? bc : bm;
        if (own > 0 && at >= first && at - own < first) { sh.bin = tid; sh.acc_c = cc; }
      }
      __syncthreads();
      const int line = sh.bin;
      const int above = static_cast<int>(sh.acc_c);
      if (quick && line >= 0 && above <= kSampleList) {
        // every block hands its tokens down to the line to block 0, whose list they share out among themselves (its order does not matter:
        // the list is sorted)
        unsigned long long* list = cluster.map_shared_rank(sh.list, 0);
        int* count = cluster.map_shared_rank(&sh.n_list, 0);
        const int n_near = sh.n_near;
        for (int e0 = 0; e0 < n_near; e0 += kSampleThreads) {
          const int e = e0 + tid;
          uint32_t key = 0;
          int jn = 0;
          if (e < n_near) {
            jn = sh.near_id[e];
            key = order_key(__uint_as_float(sm_keys[jn]) / s.temp);
          }
          const bool in = key && s.bin(key_value(key)) <= line;
          const unsigned who = __ballot_sync(0xffffffffu, in);
          int at = 0;
          if (lane == 0 && who) at = atomicAdd(count, __popc(who));
          at = __shfl_sync(0xffffffffu, at, 0) + __popc(who & ((1u << lane) - 1u));
          if (in) list[at] = (static_cast<unsigned long long>(key) << 32) | (0xffffffffu - static_cast<uint32_t>(id0 + jn));
        }
        cluster.sync();
        if (rank > 0) return;
        token = pick_from_list(sh, above, use_k ? static_cast<int>(first) : above, use_k, use_p, all_m, rp.top_p, u, s.maxp, bi);
        if (tid == 0) { out_token[out_row] = token; out_status[out_row] = kSampleOk; }
        return;
      }
      cluster.sync();                            // every block has read what is cleared now
      hist_clear(sh.hist[0]);
    }
    if (tid == 0) sh.bin = kSampleBins - 1;
    __syncthreads();
  }
#pragma unroll 4
  for (int j = tid; j < n; j += kSampleThreads) {
    uint32_t key;
    if (in_smem) {
      const int i = id0 + j;
      const float x0 = __uint_as_float(sm_keys[j]), xp = s.temp == 1.0f ? x0 : x0 / s.temp;
      const bool out = (mask && !((mask[i >> 5] >> (i & 31)) & 1u)) || (s.use_minp && !(xp >= s.thresh));
      key = out ? 0u : order_key(xp);
      sm_keys[j] = key;
    } else {
      key = s.make(j);
    }
    if (!key || flat) continue;
    const float xp = key_value(key);
    const int b = s.bin(xp);
    atomicAdd(&sh.hist[0].cnt[b], 1u);
    if (!use_k) hist_add_mass(sh.hist[0], b, mass_of(xp, s.maxp), wide);      // (with top-k the tokens in the cut give their own mass)
  }
  if (in_smem) s.keys = sm_keys;
  int line = kSampleBins - 1;
  unsigned int above = kSampleList + 1;
  unsigned long long first = 0, all_m = 0;
  if (!flat) {
    cluster.sync();
    unsigned int bc = 0;
    unsigned long long bm = 0;
    if (tid < kSampleBins) hist_total<kC>(cluster, sh.hist[0], tid, wide, bc, bm);
    const unsigned int cc = block_scan(bc, reinterpret_cast<unsigned int*>(sh.counts));
    const unsigned long long cm = block_scan(bm, sh.scan);
    if (tid == kSampleThreads - 1) { sh.acc_c = cc; sh.acc_m = cm; }
    __syncthreads();
    const unsigned int all_c = sh.acc_c;
    all_m = sh.acc_m;
    __syncthreads();
    // the first filter that applies (else the draw) says how far down the order anything can be picked
    first = use_k ? min(static_cast<unsigned long long>(rp.top_k), static_cast<unsigned long long>(all_c))
                                           : mass_target(use_p ? static_cast<double>(rp.top_p) : u, !use_p, all_m);
    if (tid < kSampleBins) {
      const unsigned long long at = use_k ? cc : cm, own = use_k ? bc : bm;
      if (own > 0 && at >= first && at - own < first) { sh.bin = tid; sh.acc_c = cc; }
    }
    __syncthreads();
    line = sh.bin;
    above = sh.acc_c;
  }
  if (above <= kSampleList) {
    // block 0 gathers in place, the others hand their shares over through its shared memory
    for (int j = tid; j < n; j += kSampleThreads) {
      const uint32_t key = s.key(j);
      if (key && s.bin(key_value(key)) <= line)
        sh.list[atomicAdd(&sh.n_list, 1)] = (static_cast<unsigned long long>(key) << 32) | (0xffffffffu - static_cast<uint32_t>(id0 + j));
    }
    cluster.sync();
    if (rank > 0) {
      int at = 0;
#pragma unroll
      for (int r = 0; r < kC; ++r)
        if (r < rank) at += *cluster.map_shared_rank(&sh.n_list, r);
      unsigned long long* dst = cluster.map_shared_rank(sh.list, 0);
      for (int j = tid; j < sh.n_list; j += kSampleThreads) dst[at + j] = sh.list[j];
    }
    cluster.sync();
    if (rank > 0) return;                      // block 0's memory is what the others wrote to; nobody reads theirs any more
    token = pick_from_list(sh, static_cast<int>(above), use_k ? static_cast<int>(first) : static_cast<int>(above), use_k, use_p, all_m, rp.top_p, u, s.maxp, bi);
  } else {
    if (!flat) cluster.sync();                 // every block has read the histograms that the descents reuse
    Cut cut{0u, 0x7fffffff};
    if (use_k) cut = select_prefix<kC>(cluster, s, cut, false, 0.0, false, rp.top_k, wide, sh);
    if (use_p) cut = select_prefix<kC>(cluster, s, cut, true, static_cast<double>(rp.top_p), false, 0, wide, sh);
    const Cut pick = select_prefix<kC>(cluster, s, cut, true, u, true, 0, wide, sh);
    token = pick.id >= 0 ? pick.id : bi;
  }
  if (rank == 0 && tid == 0) { out_token[out_row] = token; out_status[out_row] = kSampleOk; }
}

// Sample-match verification.  Rows [row_start[s], row_start[s+1]) belong to sequence s: row j holds the
// target's choice after the last committed token (j = 0) and after draft token j (j >= 1).  Draft token j
// (draft[row_start[s] + j], j < rows - 1) is accepted iff it equals selected[row j]; the first mismatch, or
// the row after the last draft, supplies the bonus token.
__global__ void accept_prefix_kernel(const int* __restrict__ selected, const int* __restrict__ draft,
                                     const int* __restrict__ row_start, int S, int* __restrict__ accepted,
                                     int* __restrict__ bonus) {
  pdl_wait();
  pdl_trigger();
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= S) return;
  const int r0 = row_start[s], n = row_start[s + 1] - r0;
  int a = 0;
  while (a < n - 1 && draft[r0 + a] == selected[r0 + a]) ++a;
  accepted[s] = a;
  bonus[s] = n > 0 ? selected[r0 + a] : -1;
}

struct SampleCall {
  const float* logits;
  int ld, V;
  const SampleRow* rows;
  const uint32_t* masks;
  int n;
  int *out_token, *out_status;
};

template <int kC>
static int launch_sample(const SampleCall& c, cudaStream_t st) {
  // a slice starts at a multiple of four tokens
  const int slice = c.V <= 0 ? 0 : kC == 1 ? c.V : static_cast<int>((static_cast<long long>(c.V) + 4 * kC - 1) / (4 * kC)) * 4;
  const size_t smem = slice <= kSampleSmemKeys ? (static_cast<size_t>(slice) + 3) / 4 * 16 : 0;      // read four keys at a time
  CAFD_CHECK_CUDA(cudaFuncSetAttribute(sample_rows_kernel<kC>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSampleSmemKeys * 4));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(c.n) * kC);
  cfg.blockDim = dim3(kSampleThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = kC;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return static_cast<int>(cudaLaunchKernelEx(&cfg, sample_rows_kernel<kC>, c.logits, c.ld, c.V, slice, c.rows, c.masks, c.out_token,
                                             c.out_status));
}

}  // namespace cafd

using namespace cafd;

// Blocks per row: eight, and fewer for a batch that would not be resident at once (two blocks to an SM) as long as a slice's keys still
// stay in shared memory beside another block's.  Clusters of a fixed eight, and one block that reads its row again in every pass, against
// this (first pass with four-byte loads), us: 256 greedy rows of 8192 41 / 16 / 11, of 32000 51 / 23 / 20; 256 rows of 8192, top-k 50 and top-p 0.95, 101 / 79 / 26.  Keys
// that don't stay in shared memory cost more than the further waves: 256 rows of 151936, top-p 0.9, 296 us with eight blocks, 555 with one.
extern "C" int cafd_sample_cluster(int n, int V, int num_sms) {
  int c = 8;
  while (c > 1 && static_cast<long long>(n) * c > 2ll * num_sms && V / (c / 2) < kSampleKeysPair) c /= 2;
  return c;
}

// rows: n 64-byte records {f32 temperature, top_p, min_p; i32 top_k; u64 seed; i64 position; i64 mask_word0;
// i32 logits_row; 20 bytes pad}.  masks: packed allowed-token bits (bit i of word i/32), or null.
extern "C" int cafd_sample_rows(const float* logits, int ld, int V, const void* rows, const uint32_t* masks, int n,
                                int* out_token, int* out_status, cafd_stream_t s) {
  if (n <= 0) return 0;
  static_assert(sizeof(SampleRow) == 64, "row record is 64 bytes");
  int dev = 0, sms = 0;
  CAFD_CHECK_CUDA(cudaGetDevice(&dev));
  CAFD_CHECK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const SampleCall c{logits, ld, V, static_cast<const SampleRow*>(rows), masks, n, out_token, out_status};
  cudaStream_t st = static_cast<cudaStream_t>(s);
  switch (cafd_sample_cluster(n, V, sms)) {
    case 8: return launch_sample<8>(c, st);
    case 4: return launch_sample<4>(c, st);
    case 2: return launch_sample<2>(c, st);
  }
  return launch_sample<1>(c, st);
}

extern "C" int cafd_accept_prefix(const int* selected, const int* draft, const int* row_start, int S, int* accepted,
                                  int* bonus, cafd_stream_t s) {
  if (S <= 0) return 0;
  launch_pdl(accept_prefix_kernel, dim3((S + 63) / 64), dim3(64), 0, static_cast<cudaStream_t>(s), selected, draft, row_start, S,
             accepted, bonus);
  return static_cast<int>(cudaGetLastError());
}
