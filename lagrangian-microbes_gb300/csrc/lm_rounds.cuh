// What the two forms of the interaction (k_rounds.cu, k_events.cu) share: the time limit, the global
// state words, and the groups of ensembles that a launch works through.
#pragma once
#include "lm_internal.h"

namespace lm {

constexpr unsigned long long ROUNDS_TIMEOUT_NS = 2000000000ull;  // 2 s

__device__ __forceinline__ unsigned long long globaltimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Vertex state words are read and written with relaxed .gpu operations: each word is the only
// shared state a pair needs, and a word changes only through the applier of its vertex's current
// pair, so coherence of the single word is all the ordering required.
__device__ __forceinline__ unsigned long long ld_relaxed(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void st_relaxed(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Groups of whole ensembles (consecutive in cell order) whose vertices fit the blocks' shared
// memory, run one after another by every block. No barrier separates the groups: pairs never join
// two ensembles, and a block that is still in group g while another has moved to g + 1 only
// delays the handoffs of g + 1 that cross into it, whose words it loads from global memory when it
// gets there (the same rule that covers blocks starting at different times).
//
// A step's groups are shared out by their entries: k_rounds_events takes those whose microbes have EV_MEAN_LO to
// EV_MEAN_HI neighbours, seen from a list entry (sum of d^2 over sum of d: dense parts count for what they hold), and
// k_rounds the others. Short lists: a ready pair is found by its owner within a pass of a few instructions, and claims
// and queues cost more than the polls saved. Very long ones: chains through the watchers last longer than the polls. Per
// launch, polled / by events, ensembles of one even density: 8 x 60k microbes at 7 neighbours 80 / 91 us, at 11 138 /
// 139, at 22 329 / 241, at 48 951 / 495, at 96 1,996 / 1,362, at 192 3,841 / 4,998. Uneven densities narrow the range: 256
// ensembles of 1e3-2e5 microbes (16 groups), fresh lattices / after 9 days of flow, polled 6.37 / 7.39 ms; events from 14
// to 64 neighbours 6.10 / 7.55, to 128 6.35 / 8.98, from 26 to 64 6.06 / 7.13, to 88 5.87 / 7.11 (but a step 16.97
// ms against 16.46), from 34 to 88 5.87 / 7.41.
// So the range is the uneven batch's: the mean cannot tell the two kinds apart, and even groups of 14 to 26 or 64 to
// 128 neighbours are polled although events are faster there.
constexpr int TL_GROUPS_MAX = 64;
constexpr unsigned long long EV_MEAN_LO = 26, EV_MEAN_HI = 64;
struct TileGroups {
  uint32_t lo[TL_GROUPS_MAX + 1];     // groups [lo[g], lo[g + 1]) of cell-order vertices, g < n
  uint32_t first[TL_GROUPS_MAX + 1];  // their ensembles [first[g], first[g + 1]) in key order
  int n;                              // 0: the step does not fit
  unsigned long long taken;           // groups that k_rounds_events takes
  unsigned long long sum[TL_GROUPS_MAX][2];
};


// The groups of a step whose blocks hold `cap` vertices together (block-uniform, in shared memory; es:
// working memory of es_cap words). Greedy: the k-th ensemble in key order, e = eord[k], holds the
// vertices from cstart[cell_base_e] to the next one's start; a group takes whole ensembles consecutive in
// that order while they fit (none when one ensemble alone is larger than cap). `shared_out`: with TileGroups::taken.
__device__ __forceinline__ void make_groups(const Bufs& b, uint32_t n_valid, uint32_t cap, uint32_t* es,
                                            uint32_t es_cap, TileGroups& tg, bool shared_out) {
  const uint32_t E = b.n_ens;
  if (n_valid <= cap) {
    if (threadIdx.x == 0) {
      tg.lo[0] = tg.first[0] = 0;
      tg.lo[1] = n_valid;
      tg.first[1] = E;
      tg.n = 1;
    }
  } else {
    const bool fits = E + 1 <= es_cap;
    if (fits) {
      for (uint32_t e = threadIdx.x; e < E; e += blockDim.x) es[e] = b.cstart[b.grids[b.eord[e]].cell_base];
      if (threadIdx.x == 0) es[E] = n_valid;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      bool ok = fits;
      int g = 0;  // the open group starts at lo[g]
      if (ok) {
        tg.lo[0] = es[0];
        tg.first[0] = 0;
      }
      for (uint32_t e = 1; e <= E && ok; ++e) {
        if (es[e] - tg.lo[g] <= cap) continue;  // ensemble e - 1 fits the open group
        if (es[e - 1] != tg.lo[g]) {            // close the group before ensemble e - 1
          if (g + 1 >= TL_GROUPS_MAX) {
            ok = false;
            break;
          }
          tg.lo[++g] = es[e - 1];
          tg.first[g] = e - 1;
        }
        ok = es[e] - tg.lo[g] <= cap;  // else ensemble e - 1 alone is larger than the blocks hold
      }
      if (ok) {
        tg.lo[g + 1] = n_valid;
        tg.first[g + 1] = E;
      }
      tg.n = ok ? g + 1 : 0;
    }
  }
  __syncthreads();
  if (!shared_out) {  // (block-uniform)
    if (threadIdx.x == 0) tg.taken = 0;
    __syncthreads();
    return;
  }
  for (int k = threadIdx.x; k < 2 * tg.n; k += blockDim.x) tg.sum[k >> 1][k & 1] = 0;
  __syncthreads();
  for (uint32_t e = threadIdx.x; tg.n && e < E; e += blockDim.x) {
    const uint32_t u = b.eord[e];
    int g = 0;
    for (int step = TL_GROUPS_MAX / 2; step; step >>= 1)
      if (g + step < tg.n && tg.first[g + step] <= e) g += step;
    atomicAdd(&tg.sum[g][0], b.edir[2 * u]);
    atomicAdd(&tg.sum[g][1], b.edir[2 * u + 1]);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long taken = 0;
    for (int g = 0; g < tg.n; ++g) {
      const unsigned long long d = tg.sum[g][0], dd = tg.sum[g][1];
      if (d && dd >= EV_MEAN_LO * d && dd <= EV_MEAN_HI * d) taken |= 1ull << g;
    }
    tg.taken = taken;
  }
  __syncthreads();
}

}  // namespace lm
