// K3: fixed-radius neighbour search over the cell-sorted particles, replacing
// cKDTree(X).query_pairs(r=interaction_radius, p=interaction_norm) (interaction_simulator.py:93-98).
//
// Distance semantics are the reference's: Minkowski-p on raw (lon, lat) degrees, inclusive
// (d <= r), on float32 positions promoted to float64. For p = 2 the decision is
// fl(fl(dx*dx) + fl(dy*dy)) <= fl(r*r) in float64 without FMA contraction; p = 1 uses |dx| + |dy| <= r
// and p = inf uses max(|dx|, |dy|) <= r. A float32 test accepts or rejects every candidate whose
// float32 distance lies outside a relative band of 2e-6 around the radius (its rounding error is
// below 3e-7 relative), and only candidates inside the band are decided in float64.
//
// One thread per particle (cell order) scans the three rows of its 3x3 cell neighbourhood; the
// three cells of a row are consecutive keys, hence one contiguous run of the sorted array. Each
// neighbour list is kept sorted by descending pair priority, the order in which the interaction
// applies pairs: lists of up to SLAB entries are gathered and ranked by k_sweep and stored in the
// per-vertex slab; longer lists are rebuilt by a second kernel into a per-step overflow area
// (allocated with an atomic cursor, regrown by the host on overflow) and put in order there.
//
// Pair priority: a 64-bit order hash of (seed, step, i, j) (the output function of SplitMix64, a
// bijection of its input, so no two pairs of a step share a priority). Any fixed order is a valid
// choice for the reference's unordered set iteration. A random order keeps the dependency chains
// of the interaction short: on the mixed lattice of the 490k workload its longest chain is
// 56-70 pairs against 80-91 for a 2x2 checkerboard-colour-major order (measured on the oracle),
// and degree-first orders are worse still (110-180).
#include <algorithm>

#include "lm_internal.h"
#include "lm_philox.cuh"

namespace lm {

__device__ __forceinline__ bool within(const PairParams& pp, float2 a, float2 b) {
  const float dx = a.x - b.x, dy = a.y - b.y;
  if (pp.norm == 2) {
    const float d2 = __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
    if (d2 < pp.r2f_lo) return true;
    if (d2 > pp.r2f_hi) return false;
    const double ddx = __dsub_rn((double)a.x, (double)b.x), ddy = __dsub_rn((double)a.y, (double)b.y);
    return __dadd_rn(__dmul_rn(ddx, ddx), __dmul_rn(ddy, ddy)) <= pp.r2;
  } else if (pp.norm == 1) {
    const float d1 = fabsf(dx) + fabsf(dy);
    if (d1 < pp.rf_lo) return true;
    if (d1 > pp.rf_hi) return false;
    const double ddx = __dsub_rn((double)a.x, (double)b.x), ddy = __dsub_rn((double)a.y, (double)b.y);
    return __dadd_rn(fabs(ddx), fabs(ddy)) <= pp.r;
  } else {
    const float di = fmaxf(fabsf(dx), fabsf(dy));
    if (di < pp.rf_lo) return true;
    if (di > pp.rf_hi) return false;
    const double ddx = __dsub_rn((double)a.x, (double)b.x), ddy = __dsub_rn((double)a.y, (double)b.y);
    return fmax(fabs(ddx), fabs(ddy)) <= pp.r;
  }
}

// The float32 side of within() without branches: the distance in the norm's terms, with the bounds below which it is
// inside the radius (lo) and above which it is outside (hi); in between within() decides.
struct Band {
  float lo, hi;
};
__device__ __forceinline__ Band band_of(const PairParams& pp) {
  return pp.norm == 2 ? Band{pp.r2f_lo, pp.r2f_hi} : Band{pp.rf_lo, pp.rf_hi};
}
__device__ __forceinline__ float norm_dist(int norm, float2 a, float2 b) {
  const float dx = a.x - b.x, dy = a.y - b.y;
  const float d2 = __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
  return norm == 2 ? d2 : norm == 1 ? fabsf(dx) + fabsf(dy) : fmaxf(fabsf(dx), fabsf(dy));
}

// The three rock-paper-scissors outcomes of pair (local ids la, lb) at `step`, as list-entry bits:
// the pair's Philox uniform (interactions.py:20's np.random.rand(), keyed by the pair) against the
// ensemble's forward-win threshold of each matchup (interactions.py:24-35), u53 < t exactly as
// r < p. Only the entry of the endpoint that applies the pair (the lower cell-order index) gets them.
__device__ __forceinline__ uint32_t win_bits(const EnsInfo& info, uint32_t la, uint32_t lb, uint32_t step) {
  const PairDraw d = pair_draw(min(la, lb), max(la, lb), step, info.seed_lo, info.seed_hi);
  return ((d.u53 < info.t_rs ? 1u : 0u) | (d.u53 < info.t_pr ? 2u : 0u) | (d.u53 < info.t_sp ? 4u : 0u))
         << ENTRY_WIN_SHIFT;
}

// a before b: higher priority first, ties by lower partner id (one global order on pairs).
__device__ __forceinline__ bool before(unsigned long long pa, uint32_t ia, unsigned long long pb, uint32_t ib) {
  return pa > pb || (pa == pb && ia < ib);
}

struct Vertex {
  uint32_t s, e, base, cx, cy;
  EnsGrid g;
  float2 ps;
};

__device__ __forceinline__ uint32_t ens_of(const Bufs& b, uint32_t s) { return b.n_ens == 1 ? 0u : b.sens[s]; }

__device__ __forceinline__ Vertex load_vertex(const Bufs& b, uint32_t s) {
  Vertex v;
  v.s = s;
  v.e = ens_of(b, s);
  v.ps = b.spos[s];
  v.g = b.grids[v.e];
  v.base = b.ens[v.e].base;
  cell_of(v.g, v.ps.x, v.ps.y, &v.cx, &v.cy);
  return v;
}

// The cell-order ranges [t0[k], t1[k]) of the (at most six) key runs of v's 3x3 neighbourhood, all cell starts loaded
// together, so a microbe waits for one round of those loads; missing runs are empty. A cell's key is a row's part
// plus a column's part, so the columns (and whether they straddle a tile edge) are worked out once for the three rows.
__device__ __forceinline__ void neighbour_runs(const Bufs& b, const Vertex& v, uint32_t* t0, uint32_t* t1) {
  const uint32_t sh = v.g.tshift, mask = (1u << sh) - 1u, ntx = tiles_x(v.g);
  const uint32_t x0 = v.cx ? v.cx - 1u : 0u, x1 = min(v.cx + 1u, (uint32_t)v.g.ncx - 1u);
  const bool two = (x0 >> sh) != (x1 >> sh);
  const uint32_t lo = ((x0 >> sh) << (2u * sh)) + (x0 & mask), hi = ((x1 >> sh) << (2u * sh)) + (x1 & mask);
  const uint32_t lo_end = two ? lo | mask : hi, hi_start = hi & ~mask;  // the edge lies between them
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    const int ry = (int)v.cy + r - 1;
    const bool row = ry >= 0 && ry < v.g.ncy;
    const uint32_t y = (uint32_t)(row ? ry : (int)v.cy);
    const uint32_t* c = b.cstart + v.g.cell_base + ((((y >> sh) * ntx) << (2u * sh)) + ((y & mask) << sh));
    t0[2 * r] = row ? c[lo] : 0u;
    t1[2 * r] = row ? c[lo_end + 1u] : 0u;
    t0[2 * r + 1] = row && two ? c[hi_start] : 0u;
    t1[2 * r + 1] = row && two ? c[hi + 1u] : 0u;
  }
}

__device__ __forceinline__ uint32_t lanemask_lt_p() {
  uint32_t m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// What a warp of k_sweep keeps: a column per lane (its neighbours, then their local ids, their outcome bits and at last
// its list), the draws in queue order as lane * SLAB + slot, and each lane's local id and ensemble.
struct SweepWarp {
  uint32_t col[SLAB][32];
  uint32_t la[32], ens[32];
  uint16_t queue[32 * SLAB];
};

// The places of the m neighbours of column `lane` by their whole priorities, four bits each.
__device__ __noinline__ uint32_t sweep_exact(const uint32_t* __restrict__ sid, const SweepWarp& sh, uint32_t lane,
                                             uint32_t m, uint32_t la, uint32_t base, unsigned long long hash) {
  uint32_t places = 0;
  for (uint32_t i = 0; i < m; ++i) {
    const uint32_t li = sid[sh.col[i][lane]] - base;
    const unsigned long long p = order_hash_from(hash, min(la, li), max(la, li));
    uint32_t k = 0;
    for (uint32_t j = 0; j < m; ++j) {
      const uint32_t lj = sid[sh.col[j][lane]] - base;
      k += before(order_hash_from(hash, min(la, lj), max(la, lj)), lj, p, li) ? 1u : 0u;
    }
    places |= k << (4 * i);
  }
  return places;
}

// Lists of up to SLAB neighbours, a microbe a thread. Bound by instruction issue and the latency of its loads, so:
//   - the candidate loop does no more than the distance test and one store of the index into the lane's column, run
//     by run (walking the six runs as one range took 5 selects a candidate: 47 us against 44 for 490,000 microbes on
//     a lattice, two candidates at a time 46, the next position loaded ahead 45);
//   - the order comes from the upper halves of the priorities: each pair of neighbours adds one to the place of the
//     later one (packed four bits each). Equal halves send a microbe to sweep_exact;
//   - the outcome draws of the warp are spread evenly over its lanes through a queue (about half the entries of a
//     lattice list need a draw, and the lanes need them at different slots);
//   - lists leave through the column as two 16-byte stores;
//   - counters are added to once per block (below).
// 53 -> 44 us for 490,000 microbes on a lattice, 64 -> 48 mixed, 211 -> 155 for 2,000,000 mixed, 142 -> 111 for 32
// ensembles of 1,200,000 in all (a sorting network over 64-bit priorities, a shift register of neighbours and two
// counters per warp before). Blocks of 128: 3-15 % slower with counters per warp; 5 blocks an SM 118 and 160 us on the
// last two, 6 the figures above.
__global__ void __launch_bounds__(SLOT_BLOCK, 6) k_sweep(Bufs b, PairParams pp, StepArgs a, Ctrl* ctrl) {
  pdl_wait();
  if (ctrl->halt) return;
  __shared__ SweepWarp sh_all[SLOT_BLOCK / 32];
  const uint32_t n_valid = ctrl->n_valid;
  const uint32_t step = a.use_ctrl_step ? ctrl->step : a.step0;
  const uint32_t s = blockIdx.x * SLOT_BLOCK + threadIdx.x, lane = threadIdx.x & 31u;
  SweepWarp& sh = sh_all[threadIdx.x >> 5];
  uint32_t m = 0, la = 0, base = 0, e = 0, id = 0;
  unsigned long long hash = 0;
  if (s < n_valid) {
    const Vertex v = load_vertex(b, s);
    const Band band = band_of(pp);
    id = b.sid[s];
    e = v.e;
    base = v.base;
    la = id - base;
    hash = order_hash_base(step, ((unsigned long long)b.ens[e].seed_hi << 32) | b.ens[e].seed_lo);
    uint32_t t0[6], t1[6];
    neighbour_runs(b, v, t0, t1);
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      for (uint32_t t = t0[q]; t < t1[q]; ++t) {
        const float2 pt = b.spos[t];
        const float dist = norm_dist(pp.norm, v.ps, pt);
        bool in = dist < band.lo;
        if (!in && !(dist > band.hi)) in = within(pp, v.ps, pt);
        if (in && t != s) {
          if (m < SLAB) sh.col[m][lane] = t;
          ++m;
        }
      }
    }
  }
  const bool is_long = m > SLAB;
  const uint32_t mk = is_long ? 0u : m;  // (longer lists are collected again by k_sweep_long)
  uint32_t nb[SLAB], key[SLAB], need = 0, places = 0;
  bool tie = false;
#pragma unroll
  for (int k = 0; k < (int)SLAB; ++k) {
    key[k] = SLAB - 1u - k;  // empty slots last
    nb[k] = 0;
    if ((uint32_t)k < mk) {
      const uint32_t t = sh.col[k][lane], lb = b.sid[t] - base;
      key[k] = (uint32_t)(order_hash_from(hash, min(la, lb), max(la, lb)) >> 32);
      tie |= key[k] < SLAB;
      nb[k] = t;
      need |= t > s ? 1u << k : 0u;  // the endpoint below in cell order applies the pair
    }
  }
  const bool few = __all_sync(0xffffffffu, mk <= 4);
  if (mk > 1) {
    // each of the first W slots against each: the one that loses moves back a place
#define LM_PLACES(W)                                              \
  _Pragma("unroll") for (int i = 0; i < W; ++i) {                 \
    _Pragma("unroll") for (int j = i + 1; j < W; ++j) {           \
      places += key[i] > key[j] ? 1u << (4 * j) : 1u << (4 * i);  \
      tie |= key[i] == key[j];                                    \
    }                                                             \
  }
    if (few) {
      LM_PLACES(4)
    } else {
      LM_PLACES(8)
    }
#undef LM_PLACES
    if (tie) places = sweep_exact(b.sid, sh, lane, mk, la, base, hash);
  }
  // the draws
  const uint32_t cnt = __popc(need);
  uint32_t incl = cnt;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= (uint32_t)o) incl += y;
  }
  const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
  uint32_t pos = incl - cnt;
#pragma unroll
  for (int k = 0; k < (int)SLAB; ++k) {
    if ((need >> k) & 1u) {
      sh.col[k][lane] = b.sid[nb[k]] - base;
      sh.queue[pos++] = (uint16_t)(lane * SLAB + k);
    }
  }
  sh.la[lane] = la;
  sh.ens[lane] = e;
  __syncwarp();
  for (uint32_t q = lane; q < total; q += 32) {
    const uint32_t src = sh.queue[q], owner = src / SLAB;
    uint32_t* slot = &sh.col[src % SLAB][owner];
    *slot = win_bits(b.ens[sh.ens[owner]], sh.la[owner], *slot, step);
  }
  __syncwarp();
  if (s < n_valid) {
    uint32_t first = NONE;
    if (mk) {
      uint32_t ent[SLAB];
#pragma unroll
      for (int k = 0; k < (int)SLAB; ++k) ent[k] = nb[k] | ((need >> k) & 1u ? sh.col[k][lane] : 0u);
#pragma unroll
      for (int k = 0; k < (int)SLAB; ++k)
        if ((uint32_t)k < mk) sh.col[(places >> (4 * k)) & 7u][lane] = ent[k];
      first = sh.col[0][lane];  // (entries past the list hold what is left there: never read)
      uint4* row = reinterpret_cast<uint4*>(b.slab + (size_t)s * SLAB);
      row[0] = make_uint4(first, sh.col[1][lane], sh.col[2][lane], sh.col[3][lane]);
      if (mk > 4) row[1] = make_uint4(sh.col[4][lane], sh.col[5][lane], sh.col[6][lane], sh.col[7][lane]);
    }
    b.deg[s] = m;
    if (b.plog) b.level[s] = 0;
    b.wstate[s] = pack_state(first, 0u, b.species[id]);  // entry 0 of the list; of long ones set by k_sweep_long
  }
  // The step's directed entries, and the list of the long ones (finished by k_sweep_long): one atomic each per block.
  // With one per warp, and a list of all microbes with pairs besides, the warps waited for the counters' line (2,000,000
  // microbes: 185 us against 168).
  __shared__ uint32_t w_dir[SLOT_BLOCK / 32], w_long[SLOT_BLOCK / 32], long_at;
  const uint32_t w = threadIdx.x >> 5, long_mask = __ballot_sync(0xffffffffu, is_long);
  const uint32_t dir = __reduce_add_sync(0xffffffffu, m);
  if (b.edir) {  // per ensemble (a warp of one ensemble, the rule in cell order, adds once), degrees of 1,023 at most
    const uint32_t m2 = min(m, 1023u), lead = __shfl_sync(0xffffffffu, e, 0);
    if (__all_sync(0xffffffffu, e == lead || m == 0u)) {
      const uint32_t sq = __reduce_add_sync(0xffffffffu, m2 * m2);
      if (lane == 0 && dir) {
        atomicAdd(b.edir + 2 * lead, (unsigned long long)dir);
        atomicAdd(b.edir + 2 * lead + 1, (unsigned long long)sq);
      }
    } else if (m) {
      atomicAdd(b.edir + 2 * e, (unsigned long long)m);
      atomicAdd(b.edir + 2 * e + 1, (unsigned long long)(m2 * m2));
    }
  }
  if (lane == 0) {
    w_dir[w] = dir;
    w_long[w] = __popc(long_mask);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long entries = 0;
    uint32_t longs = 0;
    for (int k = 0; k < (int)(SLOT_BLOCK / 32); ++k) {
      const uint32_t n = w_long[k];
      w_long[k] = longs;
      entries += w_dir[k];
      longs += n;
    }
    if (entries) atomicAdd(&ctrl->n_dir, entries);
    if (longs) long_at = atomicAdd(&ctrl->n_long, longs);
  }
  __syncthreads();
  if (is_long) b.longv[long_at + w_long[w] + __popc(long_mask & lanemask_lt_p())] = s;
}

void launch_sweep(const Bufs& b, const PairParams& pp, const StepArgs& a, Ctrl* ctrl, cudaStream_t st) {
  if (b.nslots == 0) return;
  launch_dep(k_sweep, dim3((b.nslots + SLOT_BLOCK - 1) / SLOT_BLOCK), dim3(SLOT_BLOCK), st, b, pp, a, ctrl);
}

// Count-only pair search (the clustered stress workload, whose 1e11+ pairs per step cannot be
// listed): every unordered pair within the radius is counted once, with the same cell grid and
// the same distance test as the sweep. Microbe a (cell order) takes the members of its own cell
// with a higher cell-order index and every member of its four "forward" cells: (cx+1, cy) and the
// three cells of row cy+1 (cx-1 .. cx+1, one contiguous run).
//
// Where cells hold thousands of microbes (cluster cores), most candidates are far inside the radius
// or far outside it together with their neighbours. k_count_order sorts the members of every cell
// of at least COUNT_DENSE along a Hilbert curve, k_count_boxes takes the bounding box of every 32
// consecutive microbes (a leaf), and k_count_pairs, one warp per leaf, compares boxes first: a leaf
// whose farthest corner lies inside the radius is counted at once, one whose nearest point lies
// outside is skipped, and only the others (12 % of the candidates at 13k microbes a cell) are tested
// microbe by microbe. A warp whose microbes have few candidates lets each lane walk its own runs.
// Bound by instruction issue. 3M microbes in 400 clusters (1.3e10 pairs): 13.2 ms with every
// candidate tested, 1.7 ms by leaves (ordering 0.06 ms and boxes 0.02 ms beside it).
constexpr uint32_t COUNT_THREADS = 256;
constexpr int COUNT_RUNS = 4;
constexpr uint32_t COUNT_FEW = 256;  // candidates up to which a lane walks its runs alone: box tests, a
                                     // shared tile and a few shuffles per leaf cost about as much

__device__ __forceinline__ void count_runs(const Vertex& v, const Bufs& b, uint32_t* r0, uint32_t* r1) {
  // r[0] = the rest of the own cell, r[1] = (cx+1, cy), r[2..3] = row cy+1 from cx-1 to cx+1 (one
  // or two key runs: the row may cross a tile edge); unused runs are empty
  const uint32_t kc = v.g.cell_base + cell_index(v.g, v.cx, v.cy);
  r0[0] = v.s + 1;
  r1[0] = b.cstart[kc + 1];
  for (int q = 1; q < COUNT_RUNS; ++q) r0[q] = r1[q] = 0;
  if ((int)v.cx + 1 < v.g.ncx) {
    const uint32_t ke = v.g.cell_base + cell_index(v.g, v.cx + 1, v.cy);
    r0[1] = b.cstart[ke];
    r1[1] = b.cstart[ke + 1];
  }
  if ((int)v.cy + 1 < v.g.ncy) {
    const RowRuns rr = row_runs(v.g, max((int)v.cx - 1, 0), min((int)v.cx + 1, v.g.ncx - 1), (int)v.cy + 1);
    r0[2] = b.cstart[rr.lo[0]];
    r1[2] = b.cstart[rr.hi[0] + 1];
    if (rr.n == 2) {
      r0[3] = b.cstart[rr.lo[1]];
      r1[3] = b.cstart[rr.hi[1] + 1];
    }
  }
}

// The members of every dense cell (listed in act by k_scatter) in the order of their 32 x 32 sub-cells
// along the curve: a counting sort through shared memory, one block per cell, by way of `tmp` (the
// state words, unused here). Only the positions move: counting needs no ids.
constexpr int ORDER_THREADS = 512;
constexpr uint32_t ORDER_BINS = 1024;
__global__ void __launch_bounds__(ORDER_THREADS) k_count_order(Bufs b, Ctrl* ctrl) {
  pdl_wait();
  if (ctrl->halt) return;
  __shared__ uint32_t cnt[ORDER_BINS];
  float2* tmp = reinterpret_cast<float2*>(b.wstate);
  const uint32_t n = ctrl->act_n;
  for (uint32_t q = blockIdx.x; q < n; q += gridDim.x) {
    const uint32_t key = b.act[q], c0 = b.cstart[key], c1 = b.cstart[key + 1];
    const EnsGrid g = b.grids[ens_of(b, c0)];
    uint32_t cx, cy;
    cell_coords(g, key - g.cell_base, &cx, &cy);
    const float ox = g.x0 + (float)cx * g.c, oy = g.y0 + (float)cy * g.c, scale = 32.f * g.inv_c;
    auto sub = [&](float2 p) {  // any assignment is valid, so the clamps only keep it in range
      const uint32_t x = (uint32_t)fminf(fmaxf((p.x - ox) * scale, 0.f), 31.f);
      const uint32_t y = (uint32_t)fminf(fmaxf((p.y - oy) * scale, 0.f), 31.f);
      return hilbert_place(x, y, 5);
    };
    for (uint32_t i = threadIdx.x; i < ORDER_BINS; i += ORDER_THREADS) cnt[i] = 0;
    __syncthreads();
    for (uint32_t i = c0 + threadIdx.x; i < c1; i += ORDER_THREADS) atomicAdd(&cnt[sub(b.spos[i])], 1u);
    __syncthreads();
    if (threadIdx.x < 32) {  // exclusive scan, a row of 32 counts at a time
      uint32_t run = 0;
      for (uint32_t k = threadIdx.x; k < ORDER_BINS; k += 32) {
        const uint32_t c = cnt[k];
        uint32_t incl = c;
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
          if (threadIdx.x >= (uint32_t)o) incl += y;
        }
        cnt[k] = run + incl - c;
        run += __shfl_sync(0xffffffffu, incl, 31);
      }
    }
    __syncthreads();
    for (uint32_t i = c0 + threadIdx.x; i < c1; i += ORDER_THREADS) {
      const float2 p = b.spos[i];
      tmp[c0 + atomicAdd(&cnt[sub(p)], 1u)] = p;
    }
    __syncthreads();
    for (uint32_t i = c0 + threadIdx.x; i < c1; i += ORDER_THREADS) b.spos[i] = tmp[i];
    __syncthreads();
  }
}

// Bounding box (x0, y0, x1, y1) of every leaf, kept in the slab rows (unused here).
__global__ void __launch_bounds__(COUNT_THREADS) k_count_boxes(Bufs b, Ctrl* ctrl) {
  pdl_wait();
  if (ctrl->halt || ctrl->act_n == 0) return;
  const uint32_t s = blockIdx.x * COUNT_THREADS + threadIdx.x, n = ctrl->n_valid;
  if ((s & ~31u) >= n) return;  // warp-uniform
  const float2 p = s < n ? b.spos[s] : make_float2(NAN, NAN);  // fminf and fmaxf ignore NaN
  float4 v = make_float4(p.x, p.y, p.x, p.y);
  for (int o = 16; o > 0; o >>= 1) {
    v.x = fminf(v.x, __shfl_xor_sync(0xffffffffu, v.x, o));
    v.y = fminf(v.y, __shfl_xor_sync(0xffffffffu, v.y, o));
    v.z = fmaxf(v.z, __shfl_xor_sync(0xffffffffu, v.z, o));
    v.w = fmaxf(v.w, __shfl_xor_sync(0xffffffffu, v.w, o));
  }
  if ((s & 31u) == 0) reinterpret_cast<float4*>(b.slab)[s >> 5] = v;
}

// The float32 value that the pair test of each norm compares (r^2 for p = 2, else r).
__device__ __forceinline__ float norm_value(int norm, float dx, float dy) {
  if (norm == 2) return fmaf(dx, dx, dy * dy);
  if (norm == 1) return fabsf(dx) + fabsf(dy);
  return fmaxf(fabsf(dx), fabsf(dy));
}

// Members of `tile` (32 of them, shared memory) within the radius of `me`. A value's place in the
// float32 band around the radius is a number f clamped to [0, 1]: 1 below the band, 0 above; where
// the sum of f differs from the sum of f^2, a candidate lies inside the band and the tile is
// recounted with the exact test (the same decision as within(); one fused multiply-add in d^2 is far
// inside the band). All of it runs in the FMA pipe: two compares and two adds a candidate would
// cost more issue slots.
template <int NORM>
__device__ __forceinline__ uint32_t count_tile(const PairParams& pp, float scale, float shift, float2 me,
                                               const float2* tile) {
  const float4* t4 = reinterpret_cast<const float4*>(tile);
  float f1 = 0.f, f2 = 0.f;
#pragma unroll 8
  for (int k = 0; k < 16; ++k) {
    const float4 q = t4[k];
    const float fa = __saturatef(fmaf(norm_value(NORM, me.x - q.x, me.y - q.y), scale, shift));
    const float fb = __saturatef(fmaf(norm_value(NORM, me.x - q.z, me.y - q.w), scale, shift));
    f1 += fa + fb;
    f2 = fmaf(fa, fa, fmaf(fb, fb, f2));
  }
  uint32_t c = __float2uint_rn(f1);  // (a place just below 1 may leave the sum an ulp short)
  if (f1 != f2) {
    c = 0;
    for (int k = 0; k < 32; ++k) c += within(pp, me, tile[k]) ? 1u : 0u;
  }
  return c;
}

// Pairs of the warp's microbes of one cell (lanes `grp`, consecutive) with the candidates of its runs.
template <int NORM>
__device__ __forceinline__ unsigned long long count_group(const Bufs& b, const PairParams& pp, float lo, float hi,
                                                          float2 me, uint32_t grp, uint32_t s_last, const uint32_t* r0,
                                                          const uint32_t* r1, float2* tile) {
  const uint32_t lane = threadIdx.x & 31u;
  const bool in = (grp >> lane) & 1u;
  const uint32_t members = __popc(grp);
  const float scale = -1.f / (hi - lo), shift = hi / (hi - lo);
  const float4* boxes = reinterpret_cast<const float4*>(b.slab);
  unsigned long long cnt = 0;
  // pairs inside the group
  for (uint32_t rest = grp; rest; rest &= rest - 1) {
    const int j = __ffs(rest) - 1;
    const float2 p = make_float2(__shfl_sync(0xffffffffu, me.x, j), __shfl_sync(0xffffffffu, me.y, j));
    if (in && lane < (uint32_t)j && within(pp, me, p)) ++cnt;
  }
  float4 box = in ? make_float4(me.x, me.y, me.x, me.y) : make_float4(NAN, NAN, NAN, NAN);
  for (int o = 16; o > 0; o >>= 1) {
    box.x = fminf(box.x, __shfl_xor_sync(0xffffffffu, box.x, o));
    box.y = fminf(box.y, __shfl_xor_sync(0xffffffffu, box.y, o));
    box.z = fmaxf(box.z, __shfl_xor_sync(0xffffffffu, box.z, o));
    box.w = fmaxf(box.w, __shfl_xor_sync(0xffffffffu, box.w, o));
  }
  auto points = [&](uint32_t at, uint32_t n) {  // n <= 32 candidates from `at`; the others far away
    __syncwarp();
    tile[lane] = lane < n ? b.spos[at + lane] : make_float2(INFINITY, INFINITY);
    __syncwarp();
    if (in) cnt += count_tile<NORM>(pp, scale, shift, me, tile);
  };
#pragma unroll 1
  for (int q = 0; q < COUNT_RUNS; ++q) {
    const uint32_t a = q == 0 ? s_last + 1u : r0[q], e = r1[q];
    if (a >= e) continue;  // warp-uniform
    const uint32_t head = min(e, (a + 31u) & ~31u), tail = max(head, e & ~31u);  // whole leaves in [head, tail)
    if (head > a) points(a, head - a);
    for (uint32_t l0 = head >> 5; l0 < tail >> 5; l0 += 32) {
      const uint32_t l = l0 + lane;
      bool partial = false;
      if (l < tail >> 5) {
        const float4 v = boxes[l];
        const float nx = fmaxf(0.f, fmaxf(v.x - box.z, box.x - v.z)), ny = fmaxf(0.f, fmaxf(v.y - box.w, box.y - v.w));
        const float fx = fmaxf(v.z - box.x, box.z - v.x), fy = fmaxf(v.w - box.y, box.w - v.y);
        if (norm_value(NORM, fx, fy) < lo) cnt += 32u * members;
        else partial = !(norm_value(NORM, nx, ny) > hi);
      }
      uint32_t m = __ballot_sync(0xffffffffu, partial);
      if (m) {  // the next leaf is on its way while this one is tested
        float2 next = b.spos[((l0 + __ffs(m) - 1) << 5) + lane];
        while (m) {
          __syncwarp();
          tile[lane] = next;
          __syncwarp();
          m &= m - 1;
          if (m) next = b.spos[((l0 + __ffs(m) - 1) << 5) + lane];
          if (in) cnt += count_tile<NORM>(pp, scale, shift, me, tile);
        }
      }
    }
    if (e > tail) points(tail, e - tail);
  }
  return cnt;
}

__global__ void __launch_bounds__(COUNT_THREADS) k_count_pairs(Bufs b, PairParams pp, Ctrl* ctrl) {
  pdl_wait();
  if (ctrl->halt) return;
  __shared__ __align__(16) float2 tiles[COUNT_THREADS / 32][32];
  __shared__ unsigned long long tot;
  const uint32_t n_valid = ctrl->n_valid;
  const uint32_t blk0 = blockIdx.x * COUNT_THREADS;
  if (blk0 >= n_valid) return;  // block-uniform
  if (threadIdx.x == 0) tot = 0;
  __syncthreads();
  const uint32_t s = blk0 + threadIdx.x, lane = threadIdx.x & 31u;
  const bool valid = s < n_valid;
  // the float32 band of the norm's value around the radius; radii that float32 cannot resolve have none
  const float lo = pp.norm == 2 ? pp.r2f_lo : pp.rf_lo, hi = pp.norm == 2 ? pp.r2f_hi : pp.rf_hi;
  const bool leaves = ctrl->act_n != 0 && lo > 0.f && hi < INFINITY;
  unsigned long long cnt = 0;
  Vertex v{};
  uint32_t r0[COUNT_RUNS] = {0, 0, 0, 0}, r1[COUNT_RUNS] = {0, 0, 0, 0}, key = NONE;
  if (valid) {
    v = load_vertex(b, s);
    key = v.g.cell_base + cell_index(v.g, v.cx, v.cy);
    count_runs(v, b, r0, r1);
  }
  uint32_t most = 0;
  for (int q = 0; q < COUNT_RUNS; ++q) most += r1[q] - r0[q];
  most = __reduce_max_sync(0xffffffffu, most);
  if (!leaves || most <= COUNT_FEW) {
    for (int q = 0; q < COUNT_RUNS; ++q)
      for (uint32_t t = r0[q]; t < r1[q]; ++t) cnt += within(pp, v.ps, b.spos[t]) ? 1u : 0u;
  } else {
    for (uint32_t rest = __ballot_sync(0xffffffffu, valid); rest;) {  // the warp's cells in turn
      const int first = __ffs(rest) - 1;
      const uint32_t first_key = __shfl_sync(0xffffffffu, key, first);
      const uint32_t grp = __ballot_sync(0xffffffffu, valid && key == first_key);
      uint32_t a[COUNT_RUNS], e[COUNT_RUNS];
#pragma unroll
      for (int q = 0; q < COUNT_RUNS; ++q) {
        a[q] = __shfl_sync(0xffffffffu, r0[q], first);
        e[q] = __shfl_sync(0xffffffffu, r1[q], first);
      }
      const uint32_t s_last = (s - lane) + 31u - __clz(grp);
      float2* tile = tiles[threadIdx.x >> 5];
      if (pp.norm == 2) cnt += count_group<2>(b, pp, lo, hi, v.ps, grp, s_last, a, e, tile);
      else if (pp.norm == 1) cnt += count_group<1>(b, pp, lo, hi, v.ps, grp, s_last, a, e, tile);
      else cnt += count_group<0>(b, pp, lo, hi, v.ps, grp, s_last, a, e, tile);
      rest &= ~grp;
    }
  }
  for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
  if (lane == 0 && cnt) atomicAdd(&tot, cnt);
  __syncthreads();
  if (threadIdx.x == 0 && tot) atomicAdd(&ctrl->n_dir, 2ull * tot);
}

void launch_count_pairs(const Bufs& b, const PairParams& pp, Ctrl* ctrl, int sms, cudaStream_t st) {
  if (b.nslots == 0) return;
  const unsigned blocks = (b.nslots + COUNT_THREADS - 1) / COUNT_THREADS;
  launch_dep(k_count_order, dim3(sms * 4), dim3(ORDER_THREADS), st, b, ctrl);
  launch_dep(k_count_boxes, dim3(blocks), dim3(COUNT_THREADS), st, b, ctrl);
  launch_dep(k_count_pairs, dim3(blocks), dim3(COUNT_THREADS), st, b, pp, ctrl);
}

// Long lists (more than SLAB neighbours). A warp takes batches of up to 32 of them, consecutive in cell
// order; lane k loads vertex k's cell, position, key runs and ensemble constants, so the dependent loads
// happen once per batch, and one atomic reserves the overflow space of all its batches. Then:
//   - the members of the batch that share a cell share its candidates: the 3x3 cells are read once into
//     shared memory, and each member tests them from there, 32 a pass, and gathers its neighbours with
//     ballots;
//   - the lists of several members fill one area of LONG_AREA entries, and priorities, outcome draws and
//     the order run over the area, an entry a lane, whatever the lengths of its lists. Only the entries
//     whose endpoint applies the pair (half of them) are queued for a draw;
//   - each entry's place is the number of larger keys in its list, the key being the upper 24 bits of the
//     64-bit priority over the entry's index in its list (so keys differ). An area where two entries of a
//     list agree in those 24 bits is ranked again by the whole priorities.
// Members with more than LONG_FEW neighbours or LONG_CAND candidates are done one at a time (long_alone):
// candidates from global memory, 64 a pass, and up to LONG_SMEM_MAX entries a bucket sort: the priorities
// are uniform hashes, so 256 buckets on their top 8 bits (descending) hold about d / 256 entries each, and
// an insertion sort inside each bucket by the exact order finishes it; beyond, buckets in global memory.
// Only the sorted partners are kept (the priorities were needed for the order only).
// Bound by instruction issue (76 % of the slots, 645 instructions a list of 34). A warp per list before
// took 530 us for the 447,000 lists of 32 ensembles, 245 for the 338,000 of 2,000,000 mixed microbes and 66
// for the 81,000 of 490,000; this takes 366, 132 and 40. At 6 blocks an SM (9 KB a warp) it took 438,
// 194 and 54. 10,000 microbes with 1,100 neighbours each 21.4 -> 1.0 ms (one lane sorted such lists before).
constexpr int LONG_WARPS = 4;
constexpr uint32_t LONG_SMEM_MAX = 512;
constexpr uint32_t LONG_BUCKETS = 256;

struct LongSmem {
  uint32_t key[LONG_SMEM_MAX];  // partner's local id, then the upper half of the pair's priority (gather order)
  uint32_t t[LONG_SMEM_MAX];    // list entry (partner's cell-order index + outcome bits)
  uint32_t cur[LONG_BUCKETS];
  uint16_t ord[LONG_SMEM_MAX];  // entries in list order
  uint16_t start[LONG_BUCKETS];
};

// What a warp keeps of a batch: its members, the candidates of the cell at hand and the area of lists.
constexpr uint32_t LONG_FEW = 96;    // neighbours (keys keep 7 bits for the index)
constexpr uint32_t LONG_CAND = 192;  // candidates
constexpr uint32_t LONG_AREA = 224;  // entries (with these sizes 8 blocks of 4 warps fit an SM)
struct LongArea {
  uint32_t key[LONG_AREA];  // 16-byte aligned: four keys a load
  uint32_t t[LONG_AREA];    // list entry (partner's cell-order index + outcome bits)
  uint32_t lb[LONG_AREA];   // partner's local id; then the keys in list order
  uint16_t queue[LONG_AREA];
  uint8_t own[LONG_AREA];   // member of the batch the entry belongs to (0xff: a gap)
  float2 cpos[LONG_CAND];
  uint32_t ct[LONG_CAND];
  // the members: the part of the priority's hash that its pairs share, position, index, local id, ensemble, list
  // offset in ovf, length, place in the area, species
  unsigned long long hash[32];
  float2 ps[32];
  uint32_t s[32], la[32], e[32], o[32];
  uint16_t d[32], st[32];
  int8_t sp[32];
};
union LongShared {
  LongSmem one;
  LongArea many;
};
static_assert(sizeof(LongShared) % 16 == 0, "every warp's keys are read 16 bytes at a time");

// A list that is done alone: what its pairs' priorities need.
struct LongHead {
  unsigned long long hash;  // order_hash_base
  uint32_t la, base;
};

// Does the pair with upper priority half x and entry ex come before (y, ey)? Equal halves go by the whole priority.
__device__ __forceinline__ bool long_before(const Bufs& b, const LongHead& h, uint32_t x, uint32_t ex, uint32_t y,
                                            uint32_t ey) {
  if (x != y) return x > y;
  const uint32_t lx = b.sid[entry_id(ex)] - h.base, ly = b.sid[entry_id(ey)] - h.base;
  return before(order_hash_from(h.hash, min(h.la, lx), max(h.la, lx)), lx,
                order_hash_from(h.hash, min(h.la, ly), max(h.la, ly)), ly);
}

// Exclusive scan of the counts in cur; start gets the result as well.
template <class T>
__device__ __forceinline__ void long_scan(uint32_t* cur, T* start, uint32_t lane) {
  uint32_t c[8], tot = 0;  // lane holds buckets 8 lane .. 8 lane + 7
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    c[r] = cur[8 * lane + r];
    tot += c[r];
  }
  uint32_t incl = tot;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= (uint32_t)o) incl += y;
  }
  uint32_t run = incl - tot;
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    start[8 * lane + r] = (T)run;
    cur[8 * lane + r] = run;
    run += c[r];
  }
}

// The bucket sort of entries [0, d) of sh into sh.ord (one warp).
__device__ __forceinline__ void long_sort(const Bufs& b, LongSmem& sh, const LongHead& h, uint32_t d, uint32_t lane) {
  for (uint32_t i = lane; i < LONG_BUCKETS; i += 32) sh.cur[i] = 0;
  __syncwarp();
  for (uint32_t i = lane; i < d; i += 32) atomicAdd(&sh.cur[255u - (sh.key[i] >> 24)], 1u);
  __syncwarp();
  long_scan(sh.cur, sh.start, lane);
  __syncwarp();
  for (uint32_t i = lane; i < d; i += 32) sh.ord[atomicAdd(&sh.cur[255u - (sh.key[i] >> 24)], 1u)] = (uint16_t)i;
  __syncwarp();
  for (uint32_t k = lane; k < LONG_BUCKETS; k += 32) {
    const uint32_t lo = sh.start[k], hi = sh.cur[k];
    for (uint32_t x = lo + 1; x < hi; ++x) {
      const uint16_t e = sh.ord[x];
      uint32_t y = x;
      while (y > lo && long_before(b, h, sh.key[e], sh.t[e], sh.key[sh.ord[y - 1]], sh.t[sh.ord[y - 1]])) {
        sh.ord[y] = sh.ord[y - 1];
        --y;
      }
      sh.ord[y] = e;
    }
  }
  __syncwarp();
}

// The same in global memory for the d words w = upper priority half << 32 | entry; the entries in order go to nb. Each
// entry's place in its bucket is the number of members before it. nb first holds the words' indices by bucket (20
// bits) with those places above them; the upper halves of w, free by then, take the entries at their places. Lists
// that this does not hold (2^20 entries, or 4,096 in a bucket) are put in order by one lane's heap instead.
__device__ __forceinline__ void long_sort_global(const Bufs& b, LongSmem& sh, const LongHead& h, unsigned long long* w,
                                                 uint32_t* nb, uint32_t d, uint32_t lane) {
  constexpr uint32_t IDX_BITS = 20, IDX = (1u << IDX_BITS) - 1u, MOST = (1u << (32 - IDX_BITS)) - 1u;
  uint32_t* start = sh.key;
  auto first = [&](uint32_t i, uint32_t j) {  // word i before word j?
    const unsigned long long x = w[i], y = w[j];
    return long_before(b, h, (uint32_t)(x >> 32), (uint32_t)x, (uint32_t)(y >> 32), (uint32_t)y);
  };
  for (uint32_t i = lane; i < LONG_BUCKETS; i += 32) sh.cur[i] = 0;
  __syncwarp();
  for (uint32_t i = lane; i < d; i += 32) atomicAdd(&sh.cur[255u - (uint32_t)(w[i] >> 56)], 1u);
  __syncwarp();
  long_scan(sh.cur, start, lane);
  __syncwarp();
  for (uint32_t i = lane; i < d; i += 32) nb[atomicAdd(&sh.cur[255u - (uint32_t)(w[i] >> 56)], 1u)] = i;
  __syncwarp();
  bool large = d > IDX;
  for (uint32_t k = lane; k < LONG_BUCKETS; k += 32) large |= sh.cur[k] - start[k] > MOST;
  if (__any_sync(0xffffffffu, large)) {
    if (lane == 0) {  // heap sort of the indices: the root comes last
      auto sift = [&](uint32_t root, uint32_t len) {
        for (uint32_t c = 2 * root + 1; c < len; c = 2 * root + 1) {
          if (c + 1 < len && first(nb[c], nb[c + 1])) ++c;
          if (!first(nb[root], nb[c])) break;
          const uint32_t x = nb[root];
          nb[root] = nb[c];
          nb[c] = x;
          root = c;
        }
      };
      for (uint32_t r = d / 2; r-- > 0;) sift(r, d);
      for (uint32_t end = d - 1; end > 0; --end) {
        const uint32_t x = nb[0];
        nb[0] = nb[end];
        nb[end] = x;
        sift(0, end);
      }
    }
    __syncwarp();
    for (uint32_t i = lane; i < d; i += 32) nb[i] = (uint32_t)w[nb[i]];
    __syncwarp();
    return;
  }
  for (uint32_t x = lane; x < d; x += 32) {
    const uint32_t i = nb[x] & IDX, k = 255u - (uint32_t)(w[i] >> 56);
    uint32_t place = 0;
    for (uint32_t y = start[k]; y < sh.cur[k]; ++y) {
      const uint32_t j = ((volatile uint32_t*)nb)[y] & IDX;  // (another lane may be adding its place)
      place += j != i && first(j, i) ? 1u : 0u;
    }
    ((volatile uint32_t*)nb)[x] = i | place << IDX_BITS;
  }
  __syncwarp();
  for (uint32_t k = 0, x = lane; x < d; x += 32) {
    const uint32_t i = nb[x] & IDX;
    while (sh.cur[k] <= x) ++k;  // the bucket of place x (its words' upper halves may be overwritten by now)
    reinterpret_cast<uint32_t*>(w + start[k] + (nb[x] >> IDX_BITS))[1] = reinterpret_cast<const uint32_t*>(w + i)[0];
  }
  __syncwarp();
  for (uint32_t i = lane; i < d; i += 32) nb[i] = reinterpret_cast<const uint32_t*>(w + i)[1];
  __syncwarp();
}

// One list by the whole warp, candidates from global memory: candidate i is in the run q with c[q] <= i < c[q + 1],
// which starts at t0[q].
__device__ __forceinline__ void long_alone(const Bufs& b, const PairParams& pp, uint32_t step, LongSmem& sh, uint32_t s,
                                           uint32_t d, unsigned long long o, const uint32_t (&t0)[6], const uint32_t (&c)[7]) {
  const uint32_t lane = threadIdx.x & 31u;
  const float2* __restrict__ spos = b.spos;
  const uint32_t* __restrict__ sid = b.sid;
  uint32_t* const list = b.ovf + o;
  unsigned long long* const prio = b.oprio + o;
  const Band band = band_of(pp);
  const int norm = pp.norm;
  const uint32_t id0 = sid[s];
  const EnsInfo info = b.ens[ens_of(b, s)];
  const LongHead h = {order_hash_base(step, ((unsigned long long)info.seed_hi << 32) | info.seed_lo), id0 - info.base,
                      info.base};
  const int sp = b.species[id0];
  const float2 ps = spos[s];
  const bool in_smem = d <= LONG_SMEM_MAX;
  uint32_t m = 0;
  // two slices of 32 candidates per pass, each candidate's position and id loaded together
  for (uint32_t tb = 0; tb < c[6]; tb += 64) {
    uint32_t t[2], id[2];
    float2 pt[2];
    bool in[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const uint32_t i = tb + 32u * r + lane;
      uint32_t x = t0[0] + i;
#pragma unroll
      for (int q = 1; q < 6; ++q)
        if (i >= c[q]) x = t0[q] + (i - c[q]);  // the last run starting at or before i (empty runs never win)
      t[r] = x;
      in[r] = i < c[6] && x != s;
      pt[r] = in[r] ? spos[x] : ps;
      id[r] = in[r] ? sid[x] : 0u;
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const float dist = norm_dist(norm, ps, pt[r]);
      bool ok = in[r] && dist < band.lo;
      const bool unsure = in[r] && !(dist < band.lo) && !(dist > band.hi);
      if (__any_sync(0xffffffffu, unsure) && unsure) ok = within(pp, ps, pt[r]);
      const uint32_t mask = __ballot_sync(0xffffffffu, ok);
      const uint32_t pos = m + __popc(mask & lanemask_lt_p());
      if (ok && pos < d) {  // the partner and its local id; priority and draw follow below
        if (in_smem) {
          sh.t[pos] = t[r];
          sh.key[pos] = id[r] - h.base;
        } else {
          list[pos] = t[r];
          prio[pos] = id[r] - h.base;
        }
      }
      m += __popc(mask);
    }
  }
  __syncwarp();
  // priorities and outcome draws of the d entries, one entry per lane
  for (uint32_t i = lane; i < d; i += 32) {
    const uint32_t t = in_smem ? sh.t[i] : list[i], lb = in_smem ? sh.key[i] : (uint32_t)prio[i];
    const uint32_t hi = (uint32_t)(order_hash_from(h.hash, min(h.la, lb), max(h.la, lb)) >> 32);
    const uint32_t e = t > s ? t | win_bits(info, h.la, lb, step) : t;
    if (in_smem) {
      sh.key[i] = hi;
      sh.t[i] = e;
    } else {
      prio[i] = (unsigned long long)hi << 32 | e;
    }
  }
  __syncwarp();
  if (in_smem) {
    long_sort(b, sh, h, d, lane);
    for (uint32_t i = lane; i < d; i += 32) list[i] = sh.t[sh.ord[i]];
  } else {
    long_sort_global(b, sh, h, prio, list, d, lane);
  }
  if (lane == 0) {
    list[d] = NONE;
    b.slab[(size_t)s * SLAB] = (uint32_t)o;  // a long list's overflow offset, in its unused slab row
    b.wstate[s] = pack_state(in_smem ? sh.t[sh.ord[0]] : list[0], 0u, sp);  // entry 0 of the list
  }
  __syncwarp();  // the next list reuses the shared memory
}

// A batch of up to `per` lists, lane k's the one at place q + k * next: its vertex, length, overflow offset, key runs (one
// chain of dependent loads for all of them) and cell key. `run`: the offset of the batch's first list, moved behind its last.
struct LongBatch {
  bool mine;
  uint32_t s, d, key, cand;
  unsigned long long o;
  uint32_t r0[6], len[6];
  __device__ __forceinline__ LongBatch(const Bufs& b, uint32_t q, uint32_t next, uint32_t per, uint32_t n_long,
                                       unsigned long long& run) {
    const uint32_t lane = threadIdx.x & 31u;
    mine = lane < per && q + lane * next < n_long;
    s = mine ? b.longv[q + lane * next] : 0u;
    d = mine ? b.deg[s] : 0u;
    const uint32_t room = mine ? d + 1u : 0u;
    unsigned long long incl = room;
    for (int k = 1; k < 32; k <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xffffffffu, incl, k);
      if (lane >= (uint32_t)k) incl += y;
    }
    o = run + incl - room;
    run += __shfl_sync(0xffffffffu, incl, 31);
    key = cand = 0u;
#pragma unroll
    for (int r = 0; r < 6; ++r) r0[r] = len[r] = 0u;
    if (mine) {
      const Vertex v = load_vertex(b, s);
      neighbour_runs(b, v, r0, len);
#pragma unroll
      for (int r = 0; r < 6; ++r) len[r] -= r0[r];
      key = v.g.cell_base + cell_index(v.g, v.cx, v.cy);
    }
#pragma unroll
    for (int r = 0; r < 6; ++r) cand += len[r];
  }
  // The lists that are done one at a time.
  __device__ __forceinline__ uint32_t alone() const {
    return __ballot_sync(0xffffffffu, d > LONG_FEW || cand > LONG_CAND);
  }
  // Lane k's runs as one range, in every lane.
  __device__ __forceinline__ void range(int k, uint32_t (&t0)[6], uint32_t (&c)[7]) const {
    c[0] = 0;
#pragma unroll
    for (int r = 0; r < 6; ++r) {
      t0[r] = __shfl_sync(0xffffffffu, r0[r], k);
      c[r + 1] = c[r] + __shfl_sync(0xffffffffu, len[r], k);
    }
  }
};

// The lists of a warp's batches that are done one at a time, after the others and in the same shared memory. Its own walk
// over the batches, so that neither side's registers weigh on the other. Called from the other's loop instead, with the
// runs on the stack and the kernel's parameters behind references (which the stores between two uses made it load again),
// and the ids read after the gather: 200,000 microbes with 218 neighbours each 1.33 ms, 490,000 3.23, 30,000 0.21; now 0.89,
// 2.15 and 0.14 (0.94, 2.29 and 0.15 when a warp did every list of any length by itself).
__device__ __forceinline__ void long_rest(const Bufs& b, const PairParams& pp, uint32_t step, LongSmem& sh, uint32_t first,
                                          uint32_t next, uint32_t turn, uint32_t per, uint32_t n_long,
                                          unsigned long long run) {
  __syncwarp();  // (the shared memory has been the area's)
  for (uint32_t q = first; q < n_long; q += turn) {
    const LongBatch l(b, q, next, per, n_long, run);
    for (uint32_t m = l.alone(); m; m &= m - 1) {
      const int k = __ffs(m) - 1;
      uint32_t t0[6], c[7];
      l.range(k, t0, c);
      long_alone(b, pp, step, sh, __shfl_sync(0xffffffffu, l.s, k), __shfl_sync(0xffffffffu, l.d, k),
                 __shfl_sync(0xffffffffu, l.o, k), t0, c);
    }
  }
}

// Entry i of the area at place k of its list; the first one also makes its member ready.
__device__ __forceinline__ void long_out(const Bufs& b, const LongArea& sh, uint32_t i, uint32_t v, uint32_t k) {
  const uint32_t o = sh.o[v], t = sh.t[i];
  b.ovf[(size_t)o + k] = t;
  if (k == 0) {
    const uint32_t s = sh.s[v];
    b.ovf[(size_t)o + sh.d[v]] = NONE;
    b.slab[(size_t)s * SLAB] = o;               // a long list's overflow offset, in its unused slab row
    b.wstate[s] = pack_state(t, 0u, sh.sp[v]);  // entry 0 of the list
  }
}

// The n entries of the area once more, placed by their whole priorities.
__device__ __noinline__ void long_exact(const Bufs& b, const LongArea& sh, uint32_t n) {
  for (uint32_t i = threadIdx.x & 31u; i < n; i += 32) {
    const uint32_t v = sh.own[i];
    if (v == 0xffu) continue;
    const uint32_t st = sh.st[v], end = st + sh.d[v], la = sh.la[v];
    const uint32_t base = b.ens[sh.e[v]].base, lb = b.sid[entry_id(sh.t[i])] - base;
    const unsigned long long h = sh.hash[v], p = order_hash_from(h, min(la, lb), max(la, lb));
    uint32_t k = 0;
    for (uint32_t j = st; j < end; ++j) {
      const uint32_t lj = b.sid[entry_id(sh.t[j])] - base;
      k += before(order_hash_from(h, min(la, lj), max(la, lj)), lj, p, lb) ? 1u : 0u;
    }
    long_out(b, sh, i, v, k);
  }
}

// Priorities, draws, order and output of the n entries of the area. (Not inlined, its loops not unrolled: with four
// copies of an unrolled form the warps waited on instruction fetches, 7.9 of the 14 cycles between two instructions.)
__device__ __noinline__ void long_flush(const Bufs& b, uint32_t step, LongArea& sh, uint32_t n) {
  const uint32_t lane = threadIdx.x & 31u;
  __syncwarp();
  uint32_t queued = 0;
#pragma unroll 1
  for (uint32_t i0 = 0; i0 < n; i0 += 32) {
    const uint32_t i = i0 + lane;
    const uint32_t v = i < n ? sh.own[i] : 0xffu;
    uint32_t key = 0;  // gaps between the lists stay below every entry
    bool draw = false;
    if (v != 0xffu) {
      const uint32_t t = sh.t[i], la = sh.la[v], lb = b.sid[t] - b.ens[sh.e[v]].base;
      const unsigned long long p = order_hash_from(sh.hash[v], min(la, lb), max(la, lb));
      key = ((uint32_t)(p >> 33) & ~127u) | (127u - (i - sh.st[v]));
      draw = t > sh.s[v];
      sh.lb[i] = lb;
    }
    if (i < n) sh.key[i] = key;
    const uint32_t mask = __ballot_sync(0xffffffffu, draw);
    if (draw) sh.queue[queued + __popc(mask & lanemask_lt_p())] = (uint16_t)i;
    queued += __popc(mask);
  }
  __syncwarp();
#pragma unroll 1
  for (uint32_t q = lane; q < queued; q += 32) {
    const uint32_t i = sh.queue[q], v = sh.own[i];
    sh.t[i] |= win_bits(b.ens[sh.e[v]], sh.la[v], sh.lb[i], step);
  }
  __syncwarp();
#pragma unroll 1
  for (uint32_t i = lane; i < n; i += 32) {
    const uint32_t v = sh.own[i];
    if (v == 0xffu) continue;
    const uint32_t st = sh.st[v], end = st + sh.d[v], key = sh.key[i];
    uint32_t k = 0;
#pragma unroll 1
    for (uint32_t j = st; j < end; j += 4) {  // keys have 31 bits: the difference is negative where the other is larger
      const uint4 x = *reinterpret_cast<const uint4*>(&sh.key[j]);
      k += ((key - x.x) >> 31) + ((key - x.y) >> 31) + ((key - x.z) >> 31) + ((key - x.w) >> 31);
    }
    sh.lb[st + k] = key;
    long_out(b, sh, i, v, k);
  }
  __syncwarp();
  bool tie = false;
#pragma unroll 1
  for (uint32_t i = lane; i + 1 < n; i += 32) {
    const uint32_t v = sh.own[i];
    tie |= v != 0xffu && v == sh.own[i + 1] && (sh.lb[i] ^ sh.lb[i + 1]) < 128u;
  }
  if (__any_sync(0xffffffffu, tie)) long_exact(b, sh, n);  // (about one list of 4,000 at 96 entries)
  __syncwarp();
}

__global__ void __launch_bounds__(LONG_WARPS * 32, 8) k_sweep_long(Bufs b, PairParams pp, StepArgs a, Ctrl* ctrl) {
  pdl_wait();
  if (ctrl->halt) return;
  __shared__ __align__(16) LongShared sh_all[LONG_WARPS];
  const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
  LongArea& sh = sh_all[w].many;
  const uint32_t n_long = ctrl->n_long;
  const uint32_t step = a.use_ctrl_step ? ctrl->step : a.step0;
  const unsigned long long cap = ctrl->ovf_cap;
  const Band band = band_of(pp);
  const uint32_t gw = blockIdx.x * LONG_WARPS + w, nw = gridDim.x * LONG_WARPS;
  // batches of `per` vertices, the same number for every warp as nearly as can be: this warp's are gw, gw + nw, ...
  if (n_long == 0) return;
  const uint32_t turns = (n_long + 32u * nw - 1) / (32u * nw), per = (n_long + turns * nw - 1) / (turns * nw);
  // where most lists are done one at a time, a warp's are spread over all of them instead: the longest lie together
  // (10,000 microbes with 1,100 neighbours each, ordered by one lane: 29 ms a step in order, 22 spread)
  const bool spread = ctrl->n_dir > (unsigned long long)LONG_FEW * n_long;
  const uint32_t first = spread ? gw : gw * per, next = spread ? nw : 1u, turn = nw * per;
  unsigned long long sum = 0;
  bool too_many = false;
  for (uint32_t q = first; q < n_long; q += turn) {
    if (lane >= per || q + lane * next >= n_long) continue;
    const uint32_t d = b.deg[b.longv[q + lane * next]];
    sum += d + 1u;  // the list and its end mark
    too_many |= d > MAX_DEGREE;
  }
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  too_many = __any_sync(0xffffffffu, too_many);
  unsigned long long run = 0;
  if (sum == 0) return;
  if (lane == 0) run = atomicAdd(&ctrl->ovf_used, sum);
  run = __shfl_sync(0xffffffffu, run, 0);
  if (too_many || run + sum > cap) {  // positions would not fit the state word / the area is full
    if (lane == 0) {
      ctrl->halt = 1;
      ctrl->halt_step = ctrl->step;
      atomicOr(&ctrl->err, too_many ? (uint32_t)ERRB_ROUNDCAP : (uint32_t)ERRB_OVERFLOW);
    }
    return;
  }
  const unsigned long long run0 = run;
  bool rest = false;
  for (uint32_t q = first; q < n_long; q += turn) {
    const LongBatch l(b, q, next, per, n_long, run);
    const bool mine = l.mine;
    const uint32_t s_l = l.s, nk = __popc(__ballot_sync(0xffffffffu, mine));  // (the first nk lanes)
    const uint32_t large = l.alone();
    rest |= large != 0u;
    if (mine) {
      const uint32_t id = b.sid[s_l], e = ens_of(b, s_l);
      const EnsInfo& info = b.ens[e];
      sh.hash[lane] = order_hash_base(step, ((unsigned long long)info.seed_hi << 32) | info.seed_lo);
      sh.ps[lane] = b.spos[s_l];
      sh.s[lane] = s_l;
      sh.la[lane] = id - info.base;
      sh.e[lane] = e;
      sh.o[lane] = (uint32_t)l.o;
      sh.d[lane] = (uint16_t)l.d;  // (read for the small ones only)
      sh.sp[lane] = b.species[id];
    }
    uint32_t used = 0;  // entries in the area
    for (uint32_t left = (nk == 32u ? 0xffffffffu : (1u << nk) - 1u) & ~large; left;) {
      const int lead = __ffs(left) - 1;
      const uint32_t lead_key = __shfl_sync(0xffffffffu, l.key, lead);
      uint32_t m = __ballot_sync(0xffffffffu, mine && l.key == lead_key) & left;
      left &= ~m;
      // the six runs as one candidate range: candidate i is in the run r with c[r] <= i < c[r + 1]
      uint32_t t0[6], c[7];
      l.range(lead, t0, c);
      __syncwarp();
      for (uint32_t i = lane; i < c[6]; i += 32) {
        uint32_t x = t0[0] + i;
#pragma unroll
        for (int r = 1; r < 6; ++r)
          if (i >= c[r]) x = t0[r] + (i - c[r]);  // the last run starting at or before i (empty runs never win)
        sh.cpos[i] = b.spos[x];
        sh.ct[i] = x;
      }
      const uint32_t nc = c[6];
      __syncwarp();
      for (; m; m &= m - 1) {
        const int k = __ffs(m) - 1;
        const uint32_t s = sh.s[k], d = sh.d[k], room = (d + 3u) & ~3u;
        const float2 ps = sh.ps[k];
        if (used + room > LONG_AREA) {
          long_flush(b, step, sh, used);
          used = 0;
        }
        if (lane == 0) sh.st[k] = (uint16_t)used;
        uint32_t found = 0;
        for (uint32_t i0 = 0; i0 < nc; i0 += 32) {
          const uint32_t i = i0 + lane;
          const uint32_t t = i < nc ? sh.ct[i] : s;
          const float2 pt = sh.cpos[i];
          const float dist = norm_dist(pp.norm, ps, pt);
          bool ok = t != s && dist < band.lo;
          const bool unsure = t != s && !(dist < band.lo) && !(dist > band.hi);
          if (__any_sync(0xffffffffu, unsure) && unsure) ok = within(pp, ps, pt);
          const uint32_t mask = __ballot_sync(0xffffffffu, ok);
          const uint32_t at = found + __popc(mask & lanemask_lt_p());
          if (ok && at < d) sh.t[used + at] = t;
          found += __popc(mask);
        }
        for (uint32_t i = lane; i < room; i += 32) sh.own[used + i] = i < d ? (uint8_t)k : (uint8_t)0xff;
        used += room;
      }
    }
    if (used) long_flush(b, step, sh, used);
  }
  if (rest) long_rest(b, pp, step, sh_all[w].one, first, next, turn, per, n_long, run0);
}

void launch_sweep_long(const Bufs& b, const PairParams& pp, const StepArgs& a, Ctrl* ctrl, int sms,
                       int blocks_per_sm, cudaStream_t st) {
  // at most 8 blocks of 27 KB fit an SM's shared memory; more queue behind them
  launch_dep(k_sweep_long, dim3(sms * blocks_per_sm), dim3(LONG_WARPS * 32), st, b, pp, a, ctrl);
}

// ---- the pairs of a query, written out in (i, j) order ----
//
// The lists hold every pair at both endpoints, in priority order and cell-order indices. The pair
// (i, j), i < j, is written by the list of i: how many partners of i lie above it (k_pair_counts),
// their prefix sums (launch_scan), then each list's partners above i at their rank (k_pair_rows). A
// thread does a slab list in registers; a warp does a longer one through shared memory, or, past
// PAIR_SMEM partners, through the list's sort keys, which are free by then. On the host the same took
// 21 ms for the 4.6e5 pairs of 150k microbes (copies of all lists, a gather and a sort); the two kernels
// and the scan take 40 us (a call 21.9 -> 0.53 ms).
constexpr int PAIR_WARPS = 4;
constexpr uint32_t PAIR_SMEM = 512;

__device__ __forceinline__ uint32_t long_entry_id(const Bufs& b, size_t o, uint32_t k) {
  return b.sid[entry_id(b.ovf[o + k])];
}

__global__ void __launch_bounds__(SLOT_BLOCK) k_pair_counts(Bufs b, uint32_t n_valid, uint32_t* __restrict__ cnt) {
  const uint32_t s = blockIdx.x * SLOT_BLOCK + threadIdx.x;
  if (s >= n_valid) return;
  const uint32_t d = b.deg[s];
  if (d > SLAB) return;
  const uint32_t i = b.sid[s];
  uint32_t c = 0;
  for (uint32_t k = 0; k < d; ++k) c += b.sid[entry_id(b.slab[(size_t)s * SLAB + k])] > i ? 1u : 0u;
  cnt[i] = c;
}

__global__ void __launch_bounds__(PAIR_WARPS * 32) k_pair_counts_long(Bufs b, uint32_t n_long,
                                                                      uint32_t* __restrict__ cnt) {
  const uint32_t lane = threadIdx.x & 31u, nw = gridDim.x * PAIR_WARPS;
  for (uint32_t q = blockIdx.x * PAIR_WARPS + (threadIdx.x >> 5); q < n_long; q += nw) {
    const uint32_t s = b.longv[q], d = b.deg[s], i = b.sid[s];
    const size_t o = b.slab[(size_t)s * SLAB];
    uint32_t c = 0;
    for (uint32_t k = lane; k < d; k += 32) c += long_entry_id(b, o, k) > i ? 1u : 0u;
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0) cnt[i] = c;
  }
}

__global__ void __launch_bounds__(SLOT_BLOCK) k_pair_rows(Bufs b, uint32_t n_valid, const uint32_t* __restrict__ off,
                                                          int32_t* __restrict__ pi, int32_t* __restrict__ pj) {
  const uint32_t s = blockIdx.x * SLOT_BLOCK + threadIdx.x;
  if (s >= n_valid) return;
  const uint32_t d = b.deg[s];
  if (d > SLAB || d == 0) return;
  const uint32_t i = b.sid[s], at = off[i];
  uint32_t j[SLAB];
#pragma unroll
  for (int k = 0; k < (int)SLAB; ++k) j[k] = (uint32_t)k < d ? b.sid[entry_id(b.slab[(size_t)s * SLAB + k])] : 0u;
#pragma unroll
  for (int k = 0; k < (int)SLAB; ++k) {
    if ((uint32_t)k >= d || j[k] <= i) continue;
    uint32_t r = at;  // partners between i and j[k] come first (absent ones are 0, never above i)
#pragma unroll
    for (int q = 0; q < (int)SLAB; ++q) r += j[q] > i && j[q] < j[k] ? 1u : 0u;
    pi[r] = (int32_t)i;
    pj[r] = (int32_t)j[k];
  }
}

__global__ void __launch_bounds__(PAIR_WARPS * 32) k_pair_rows_long(Bufs b, uint32_t n_long,
                                                                    const uint32_t* __restrict__ off,
                                                                    int32_t* __restrict__ pi,
                                                                    int32_t* __restrict__ pj) {
  __shared__ uint32_t sh[PAIR_WARPS][PAIR_SMEM];
  const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5, nw = gridDim.x * PAIR_WARPS;
  for (uint32_t q = blockIdx.x * PAIR_WARPS + w; q < n_long; q += nw) {
    const uint32_t s = b.longv[q], d = b.deg[s], i = b.sid[s], at = off[i];
    const size_t o = b.slab[(size_t)s * SLAB];
    const bool in_smem = d <= PAIR_SMEM;
    uint32_t* row = in_smem ? sh[w] : reinterpret_cast<uint32_t*>(b.oprio + o);
    __syncwarp();
    uint32_t m = 0;  // the partners above i, in list order
    for (uint32_t k0 = 0; k0 < d; k0 += 32) {
      const uint32_t k = k0 + lane, j = k < d ? long_entry_id(b, o, k) : 0u;
      const uint32_t mask = __ballot_sync(0xffffffffu, k < d && j > i);
      if ((mask >> lane) & 1u) row[m + __popc(mask & lanemask_lt_p())] = j;
      m += __popc(mask);
    }
    __syncwarp();
    for (uint32_t k = lane; k < m; k += 32) {
      const uint32_t j = row[k];
      uint32_t r = at;
      for (uint32_t e = 0; e < m; ++e) r += row[e] < j ? 1u : 0u;
      pi[r] = (int32_t)i;
      pj[r] = (int32_t)j;
    }
  }
}

void launch_pair_counts(const Bufs& b, uint32_t n_valid, uint32_t n_long, uint32_t* cnt, int sms, cudaStream_t st) {
  if (n_valid) k_pair_counts<<<(n_valid + SLOT_BLOCK - 1) / SLOT_BLOCK, SLOT_BLOCK, 0, st>>>(b, n_valid, cnt);
  const unsigned blocks = std::min((n_long + PAIR_WARPS - 1) / PAIR_WARPS, (uint32_t)sms * 16u);
  if (n_long) k_pair_counts_long<<<blocks, PAIR_WARPS * 32, 0, st>>>(b, n_long, cnt);
}

void launch_pair_rows(const Bufs& b, uint32_t n_valid, uint32_t n_long, const uint32_t* off, int32_t* pi, int32_t* pj,
                      int sms, cudaStream_t st) {
  if (n_valid) k_pair_rows<<<(n_valid + SLOT_BLOCK - 1) / SLOT_BLOCK, SLOT_BLOCK, 0, st>>>(b, n_valid, off, pi, pj);
  const unsigned blocks = std::min((n_long + PAIR_WARPS - 1) / PAIR_WARPS, (uint32_t)sms * 16u);
  if (n_long) k_pair_rows_long<<<blocks, PAIR_WARPS * 32, 0, st>>>(b, n_long, off, pi, pj);
}

}  // namespace lm
