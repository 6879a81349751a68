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
constexpr int TL_GROUPS_MAX = 64;
struct TileGroups {
  uint32_t lo[TL_GROUPS_MAX + 1];     // groups [lo[g], lo[g + 1]) of cell-order vertices, g < n
  uint32_t first[TL_GROUPS_MAX + 1];  // their ensembles [first[g], first[g + 1]) in key order
  int n;                              // 0: the step does not fit
};


// The groups of a step whose blocks hold `cap` vertices together (block-uniform, in shared memory; es:
// working memory of es_cap words). Greedy: the k-th ensemble in key order, e = eord[k], holds the
// vertices from cstart[cell_base_e] to the next one's start; a group takes whole ensembles consecutive in
// that order while they fit (none when one ensemble alone is larger than cap).
__device__ __forceinline__ void make_groups(const Bufs& b, uint32_t n_valid, uint32_t cap, uint32_t* es,
                                            uint32_t es_cap, TileGroups& tg) {
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
}

}  // namespace lm
