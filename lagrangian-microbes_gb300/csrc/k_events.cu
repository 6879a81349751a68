// K4 + K5 for dense batches: the interaction of k_rounds.cu worked off by events instead of polls.
//
// As there, a block owns a contiguous range of cell-ordered vertices (a compact 2D patch) and keeps
// their states and list entries in shared memory. Nobody polls for the pairs inside a block: whoever
// advances a vertex looks at its next partner's word, and when the two name each other the pair is
// ready. Both endpoints may be advanced at the same time and see each other, so a ready pair is claimed
// first (a bit of the lower endpoint's word, set by compare-and-swap). The lane that found it goes on
// with it, or puts its lower endpoint into the block's queue, from which lanes without a pair take theirs.
//
// A vertex of the block is a 64-bit word: its current list entry (partner and outcome bits) and, in the
// upper half, its species class (its species, 0 for values outside 1..3, which neither change nor change
// others), the claim bit, whether its list is long, and its position there. The next three entries of
// a long list are prefetched into its row.
//
// A pair that crosses blocks goes through the global state words, in the hands of the block's watcher
// warps, one waiting vertex per lane. The upper endpoint is published there. The owner of the lower
// endpoint waits until that word names it, applies the pair and writes the word back with the partner
// left open (PENDING); the owner of the upper endpoint waits for that and looks up the next partner in
// its own lists. Only the applier of a vertex's current pair writes its word.
//
// Bound by the dependency chains and by issue: a dependent pair waits for one pass of a worker warp (some
// 250 instructions), one across blocks for two L2 round trips.
//
// Batches of ensembles of at least EV_SLOTS microbes launch this kernel (other contexts save the launch), and it takes
// the groups of TileGroups::taken. 32 ensembles of 1e3-2e5 microbes on 0.5-3 degrees: 1,108 us polled, 636 shared out (of which 548 here).
#include "lm_rounds.cuh"

namespace lm {

static_assert(SLAB == 8, "a list row holds a slab's entries, or an offset and three prefetched entries");
constexpr uint32_t EV_VMAX = 2048;     // vertices per block at most
constexpr uint32_t EV_VMIN = 128;      // and at least, while there are that many: fewer have most of their
                                       // pairs across blocks
constexpr size_t EV_SMEM = EV_VMAX * (8 + 4 * SLAB + 2 + 2);  // words, rows, two queues
constexpr int EV_THREADS = 512;
constexpr uint32_t EV_WATCHERS = 8;    // watcher warps of a block
constexpr uint32_t PENDING = 0xfffffffeu;  // a global word's partner: the owner looks it up (no valid entry)
constexpr uint32_t EV_CLAIM = 1u << 29, EV_LONG = 1u << 28, EV_POS = MAX_DEGREE;  // fields of the upper half
constexpr uint32_t EV_EMPTY = 0xffffu;

__device__ __forceinline__ uint32_t ev_class(int species) { return species >= 1 && species <= 3 ? (uint32_t)species : 0u; }
__device__ __forceinline__ unsigned long long ev_word(uint32_t species, uint32_t is_long, uint32_t pos, uint32_t entry) {
  return (unsigned long long)((species << 30) | is_long | pos) << 32 | entry;
}
__device__ __forceinline__ uint32_t hi32(unsigned long long w) { return (uint32_t)(w >> 32); }

// Shared memory by 32-bit address. The words that several warps of a block write are read and written
// as volatile.
__device__ __forceinline__ uint32_t lds(uint32_t a) {
  uint32_t v;
  asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t lds16(uint32_t a) {
  uint16_t v;
  asm volatile("ld.volatile.shared.u16 %0, [%1];" : "=h"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long lds64(uint32_t a) {
  unsigned long long v;
  asm volatile("ld.volatile.shared.u64 %0, [%1];" : "=l"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void sts(uint32_t a, uint32_t v) {
  asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void sts64(uint32_t a, unsigned long long v) {
  asm volatile("st.volatile.shared.u64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
}
__device__ __forceinline__ void sts16(uint32_t a, uint32_t v) {
  asm volatile("st.volatile.shared.u16 [%0], %1;" ::"r"(a), "h"((uint16_t)v) : "memory");
}
__device__ __forceinline__ uint32_t atoms_add(uint32_t a, uint32_t v) {
  uint32_t r;
  asm volatile("atom.shared.add.u32 %0, [%1], %2;" : "=r"(r) : "r"(a), "r"(v) : "memory");
  return r;
}
__device__ __forceinline__ uint32_t atoms_cas(uint32_t a, uint32_t c, uint32_t v) {
  uint32_t r;
  asm volatile("atom.shared.cas.b32 %0, [%1], %2, %3;" : "=r"(r) : "r"(a), "r"(c), "r"(v) : "memory");
  return r;
}

// The class that a vertex of class a holds after a pair with one of class b and outcome bits win
// (rps_outcome, which is symmetric in the two).
__device__ __forceinline__ uint32_t ev_outcome(uint32_t a, uint32_t b, uint32_t win) {
  // 2 bits per (a, b), a * 4 + b: the forward winner (the one of the two that beats the other) and the
  // matchup {1,3} -> 0, {1,2} -> 1, {2,3} -> 2
  constexpr uint32_t FWD = (1u << 10) | (2u << 12) | (1u << 14) | (2u << 18) | (2u << 20) | (3u << 22) | (1u << 26) |
                           (3u << 28) | (3u << 30);
  constexpr uint32_t CASE = (1u << 12) | (0u << 14) | (1u << 18) | (2u << 22) | (0u << 26) | (2u << 28);
  const uint32_t k = 8u * a + 2u * b;
  const uint32_t fwd = (FWD >> k) & 3u, c = (CASE >> k) & 3u;
  const uint32_t w = (win >> c) & 1u ? fwd : a ^ b ^ fwd;  // a == b: either way a
  return a != 0u && b != 0u ? w : a;
}

struct Tile {
  // shared-memory addresses
  uint32_t w;      // [EV_VMAX] words
  uint32_t row;    // [EV_VMAX][8] a slab list's entries (NONE past the last); of a longer list its offset in
                   // ovf, and (entry, position) of three positions ahead, position p in pair 1 + p % 3
  uint32_t ready;  // [EV_VMAX] 16-bit: queue of the lower endpoints of ready pairs ...
  uint32_t cross;  // [EV_VMAX] 16-bit: ... and of the vertices whose partner is outside
  uint32_t ctl;    // TileCtl
  uint32_t lo, n;  // first vertex and vertices of the block
  __device__ __forceinline__ uint32_t word(uint32_t l) const { return w + 8u * l; }
  __device__ __forceinline__ uint32_t list(uint32_t l) const { return row + 4u * SLAB * l; }
};
// Ends of the two queues, vertices whose list is done, and the stop flag of a timeout.
enum TileCtl : uint32_t { TC_READY = 0, TC_CROSS = 8, TC_DONE = 16, TC_STOP = 20, TC_BYTES = 24 };

// A queue holds every vertex at most once, so EV_VMAX slots never overflow; a slot is EV_EMPTY until its
// vertex is written, and again after it is taken. A vertex off the queue for each lane in `mask` while
// there are any, NONE for the others (whole warp).
__device__ __forceinline__ uint32_t queue_pop(uint32_t slots, uint32_t ends, uint32_t mask) {
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t h = 0, n = 0;
  if (lane == 0) {
    const unsigned long long e = lds64(ends);
    h = (uint32_t)e;
    n = min((uint32_t)__popc(mask), (uint32_t)(e >> 32) - h);
    if (n && atoms_cas(ends, h, h + n) != h) n = 0;  // another warp was first: on the next pass
  }
  n = __shfl_sync(0xffffffffu, n, 0);
  if (n == 0) return NONE;
  h = __shfl_sync(0xffffffffu, h, 0);
  const uint32_t rank = __popc(mask & ((1u << lane) - 1u));
  if (!((mask >> lane) & 1u) || rank >= n) return NONE;
  const uint32_t p = slots + 2u * ((h + rank) & (EV_VMAX - 1));
  uint32_t v = lds16(p);
  // counted, so it is being written: a warp stores its slots right after it has reserved them. (The
  // limit only keeps the wait finite; a vertex lost to it would show as the step's timeout.)
  for (int k = 0; v == EV_EMPTY && k < (1 << 20); ++k) v = lds16(p);
  if (v == EV_EMPTY) return NONE;
  sts16(p, EV_EMPTY);
  return v;
}

// The lanes in `ready` append low to the ready queue and those in `out` append x to the queue of crossing
// vertices, and `done` more vertices are done: one atomic instruction, a counter per lane (whole warp,
// the masks and the count the same in every lane).
__device__ __forceinline__ void ev_push(const Tile& t, uint32_t ready, uint32_t low, uint32_t out, uint32_t x,
                                        uint32_t done) {
  const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
  const uint32_t add = lane == 0 ? __popc(ready) : lane == 1 ? __popc(out) : lane == 2 ? done : 0u;
  uint32_t old = 0;
  if (add) old = atoms_add(t.ctl + (lane == 0 ? TC_READY + 4u : lane == 1 ? TC_CROSS + 4u : (uint32_t)TC_DONE), add);
  const uint32_t at = __shfl_sync(0xffffffffu, old, 0) + __popc(ready & lt);
  const uint32_t to = __shfl_sync(0xffffffffu, old, 1) + __popc(out & lt);
  if ((ready >> lane) & 1u) sts16(t.ready + 2u * (at & (EV_VMAX - 1)), low);
  if ((out >> lane) & 1u) sts16(t.cross + 2u * (to & (EV_VMAX - 1)), x);
}

// Is the block done, or stopped? Every lane gets lane 0's answer.
__device__ __forceinline__ bool ev_over(const Tile& t) {
  uint32_t o = 0;
  if ((threadIdx.x & 31u) == 0) o = lds(t.ctl + TC_DONE) >= t.n || lds(t.ctl + TC_STOP) ? 1u : 0u;
  return __shfl_sync(0xffffffffu, o, 0) != 0u;
}
// Stop the block after the time limit (now and then; one lane asks).
__device__ __forceinline__ void ev_time(const Tile& t, Ctrl* ctrl, unsigned long long t0) {
  if ((threadIdx.x & 31u) == 0 && globaltimer() - t0 > ROUNDS_TIMEOUT_NS) {
    sts(t.ctl + TC_STOP, 1u);
    atomicOr(&ctrl->err, (uint32_t)ERRB_TIMEOUT);
  }
}

// Entry h >= 1 of a vertex whose entry h - 1 was not the end: as a slab list's, e = row entry h & 7, or as a
// long one's, q = its prefetched pair h % 3 (both are read before it is known which one counts). An entry
// of a long list that is not there yet comes from the list itself (its end is marked, so h is inside).
__device__ __forceinline__ uint32_t long_pair(const Tile& t, uint32_t l, uint32_t h) { return t.list(l) + 8u + 8u * (h % 3u); }
__device__ __forceinline__ uint32_t ev_entry(const Bufs& b, const Tile& t, uint32_t l, uint32_t is_long, uint32_t h,
                                             bool act) {
  const uint32_t e = lds(t.list(l) + 4u * (h & 7u));
  const unsigned long long q = lds64(long_pair(t, l, h));
  if (act && is_long && hi32(q) != h) return b.ovf[(size_t)lds(t.list(l)) + h];
  return is_long ? (uint32_t)q : h < SLAB ? e : NONE;
}

// A vertex has moved on to position h of a long list: position h + 3 takes the place of position h. The
// load is issued here and stored by the lane's next pass, about when it has arrived.
struct Prefetch {
  uint32_t l, pos, entry;  // l: NONE for nothing
};
__device__ __forceinline__ void prefetch_issue(const Bufs& b, const Tile& t, uint32_t l, uint32_t h, Prefetch& p) {
  const unsigned long long before = lds64(long_pair(t, l, h + 2u));  // the end is marked, nothing follows it
  if (hi32(before) == h + 2u ? (uint32_t)before == NONE : h + 3u > b.deg[t.lo + l]) return;
  p.l = l;
  p.pos = h + 3u;
  p.entry = b.ovf[(size_t)lds(t.list(l)) + h + 3u];
}
__device__ __forceinline__ void prefetch_store(const Tile& t, Prefetch& p) {
  if (p.l == NONE) return;
  sts64(long_pair(t, p.l, p.pos), (unsigned long long)p.pos << 32 | p.entry);
  p.l = NONE;
}

// Vertex l has just taken word nw: claim the pair with its new partner if that names l (true; *low is the
// lower endpoint), publish l if it is the upper endpoint of a pair across blocks.
__device__ __forceinline__ bool ev_meet(const Bufs& b, const Tile& t, uint32_t l, unsigned long long nw, bool act,
                                        uint32_t* low) {
  const uint32_t entry = (uint32_t)nw, y = entry_id(entry) - t.lo;
  const bool in = act && y < t.n;  // (NONE is outside, too)
  const unsigned long long wy = lds64(t.word(in ? y : 0u));
  *low = min(l, y);
  const uint32_t seen = hi32(l < y ? nw : wy);
  bool got = false;
  if (in && entry_id((uint32_t)wy) == t.lo + l && !(seen & EV_CLAIM))
    got = atoms_cas(t.word(*low) + 4u, seen, seen | EV_CLAIM) == seen;
  if (act && !in && entry != NONE && t.lo + l > entry_id(entry))
    st_relaxed(b.wstate + t.lo + l, pack_state(entry, hi32(nw) & EV_POS, (int)(hi32(nw) >> 30)));
  return got;
}

// Worker warps. Every lane applies one ready pair a pass and goes on with a pair that this made ready; a
// second one goes into the block's queue, from which lanes without a pair take theirs.
__device__ __forceinline__ void ev_work(const Bufs& b, const Tile& t, Ctrl* ctrl, unsigned long long t0) {
  Prefetch ps = {NONE, 0u, 0u}, pu = {NONE, 0u, 0u};
  uint32_t polls = 0, l = NONE;  // the lower endpoint of the lane's pair
  for (;;) {
    uint32_t empty = __ballot_sync(0xffffffffu, l == NONE);
    if (__popc(empty) >= 16) {
      const uint32_t x = queue_pop(t.ready, t.ctl + TC_READY, empty);
      if (l == NONE) l = x;
      empty = __ballot_sync(0xffffffffu, l == NONE);
    }
    prefetch_store(t, ps);
    prefetch_store(t, pu);
    if (empty == 0xffffffffu) {
      if (ev_over(t)) return;
      if ((++polls & 255u) == 0u) ev_time(t, ctrl, t0);
      continue;
    }
    const bool act = l != NONE;
    const uint32_t s = act ? l : 0u;
    const unsigned long long ws = lds64(t.word(s));
    const uint32_t u = act ? entry_id((uint32_t)ws) - t.lo : 0u;
    const unsigned long long wu = lds64(t.word(u));
    const uint32_t hs = (hi32(ws) & EV_POS) + 1u, hu = (hi32(wu) & EV_POS) + 1u;
    const uint32_t ls = hi32(ws) & EV_LONG, lu = hi32(wu) & EV_LONG;
    const uint32_t ns = ev_entry(b, t, s, ls, hs, act), nu = ev_entry(b, t, u, lu, hu, act);
    const uint32_t cs = hi32(ws) >> 30, cu = hi32(wu) >> 30, win = (uint32_t)ws >> ENTRY_WIN_SHIFT;
    const unsigned long long nws = ev_word(ev_outcome(cs, cu, win), ls, hs, ns);
    const unsigned long long nwu = ev_word(ev_outcome(cu, cs, win), lu, hu, nu);
    if (act) {
      sts64(t.word(u), nwu);
      sts64(t.word(s), nws);
    }
    __threadfence_block();  // both words before either partner's is read
    uint32_t low_s, low_u;
    const bool r_s = ev_meet(b, t, s, nws, act, &low_s), r_u = ev_meet(b, t, u, nwu, act, &low_u);
    if (act && (ls | lu)) {
      if (ls) prefetch_issue(b, t, s, hs, ps);
      if (lu) prefetch_issue(b, t, u, hu, pu);
    }
    const uint32_t more = __ballot_sync(0xffffffffu, r_s && r_u);
    const uint32_t fin = __popc(__ballot_sync(0xffffffffu, act && ns == NONE)) + __popc(__ballot_sync(0xffffffffu, act && nu == NONE));
    const uint32_t xs = __ballot_sync(0xffffffffu, act && ns != NONE && entry_id(ns) - t.lo >= t.n);
    const uint32_t xu = __ballot_sync(0xffffffffu, act && nu != NONE && entry_id(nu) - t.lo >= t.n);
    if (more | fin | xs) ev_push(t, more, low_u, xs, s, fin);
    if (xu) ev_push(t, 0u, 0u, xu, u, 0u);
    l = r_s ? low_s : r_u ? low_u : NONE;
  }
}

// Watcher warps: every lane holds one vertex that waits for a pair across blocks. When more wait than
// lanes, a vertex that is not through goes back to the end of the queue.
__device__ __forceinline__ void ev_watch(const Bufs& b, const Tile& t, Ctrl* ctrl, unsigned long long t0) {
  uint32_t l = NONE, polls = 0;
  unsigned long long w = 0;  // the vertex and its word
  Prefetch pf = {NONE, 0u, 0u};
  for (;;) {
    const uint32_t empty = __ballot_sync(0xffffffffu, l == NONE);
    if (empty) {
      const uint32_t x = queue_pop(t.cross, t.ctl + TC_CROSS, empty);
      if (l == NONE && x != NONE) {
        l = x;
        w = lds64(t.word(x));
      }
      if (!__any_sync(0xffffffffu, l != NONE)) {
        prefetch_store(t, pf);
        if (ev_over(t)) return;
        if ((++polls & 63u) == 0u) ev_time(t, ctrl, t0);
        __nanosleep(100);
        continue;
      }
    }
    const uint32_t s = t.lo + l, u = entry_id((uint32_t)w);
    unsigned long long g = 0;
    if (l != NONE) g = ld_relaxed(b.wstate + max(s, u));  // the upper endpoint's word
    prefetch_store(t, pf);
    if ((++polls & 63u) == 0u) {
      ev_time(t, ctrl, t0);
      if (ev_over(t)) return;  // (stopped: the block is not done while a vertex is held)
    }
    const uint32_t mine = l, h = (hi32(w) & EV_POS) + 1u;
    const bool moved = l != NONE && (s < u ? entry_id(state_partner(g)) == s : state_pos(g) == h);
    bool ready = false;
    uint32_t low = 0, back = 0, next = 0;
    if (moved) {
      const uint32_t lg = hi32(w) & EV_LONG, theirs = ev_class(state_species(g));
      uint32_t sp = theirs;  // (an upper endpoint: the other block has applied the pair)
      if (s < u) {           // this block applies it
        const uint32_t own = hi32(w) >> 30, win = (uint32_t)w >> ENTRY_WIN_SHIFT;
        sp = ev_outcome(own, theirs, win);
        st_relaxed(b.wstate + u, pack_state(PENDING, state_pos(g) + 1u, (int)ev_outcome(theirs, own, win)));
      }
      next = ev_entry(b, t, l, lg, h, true);
      w = ev_word(sp, lg, h, next);
      sts64(t.word(l), w);
      __threadfence_block();
      ready = ev_meet(b, t, l, w, true, &low);
      if (lg) prefetch_issue(b, t, l, h, pf);
      if (next == NONE || entry_id(next) - t.lo < t.n) l = NONE;  // else it is held on
    }
    const uint32_t rdy = __ballot_sync(0xffffffffu, ready), fin = __popc(__ballot_sync(0xffffffffu, moved && next == NONE));
    if (!__any_sync(0xffffffffu, l == NONE)) {
      const unsigned long long e = lds64(t.ctl + TC_CROSS);
      if (__shfl_sync(0xffffffffu, (uint32_t)e != hi32(e) ? 1u : 0u, 0)) {  // others wait
        back = __ballot_sync(0xffffffffu, !moved);
        if (!moved) l = NONE;
      }
    }
    if (rdy | fin | back) ev_push(t, rdy, low, back, mine, fin);
  }
}

// The pairs among cell-order vertices [g_lo, g_hi) (a group of whole ensembles, so no pair leaves it), at
// most EV_VMAX per block: every block owns an equal share, in whole warps and at least EV_VMIN. (Shares
// by the ensembles' expected pairs instead gave nothing: 636 against 650 us on the batch above.)
__device__ void ev_group(const Bufs& b, Ctrl* ctrl, unsigned long long t0, uint32_t g_lo, uint32_t g_hi) {
  extern __shared__ unsigned long long ev_raw[];
  __shared__ __align__(8) uint32_t ctl[TC_BYTES / 4];
  uint4* const rows = reinterpret_cast<uint4*>(ev_raw);  // two per vertex
  unsigned long long* const words = reinterpret_cast<unsigned long long*>(rows + 2 * EV_VMAX);
  uint32_t* const queues = reinterpret_cast<uint32_t*>(words + EV_VMAX);  // both, two slots a word
  auto sh = [](const void* p) { return (uint32_t)__cvta_generic_to_shared(p); };
  Tile t;
  t.row = sh(rows);
  t.w = sh(words);
  t.ready = sh(queues);
  t.cross = t.ready + 2u * EV_VMAX;
  t.ctl = sh(ctl);
  const uint32_t V = min(EV_VMAX, max(EV_VMIN, (((g_hi - g_lo + gridDim.x - 1) / gridDim.x) + 31u) & ~31u));
  t.lo = min(g_hi, g_lo + blockIdx.x * V);
  t.n = min(g_hi, t.lo + V) - t.lo;
  if (t.n == 0) return;  // block-uniform
  if (threadIdx.x < TC_BYTES / 4) ctl[threadIdx.x] = 0u;
  for (uint32_t l = threadIdx.x; l < EV_VMAX; l += EV_THREADS) queues[l] = 0xffffffffu;
  // the loads of a vertex are independent: the whole slab row (slot 0 of a long list is its overflow
  // offset), whatever the degree
#pragma unroll 2
  for (uint32_t l = threadIdx.x; l < t.n; l += EV_THREADS) {
    const uint32_t s = t.lo + l;
    const unsigned long long w0 = ld_relaxed(b.wstate + s);  // as the sweep left it, or a remote applier since
    const uint32_t d = b.deg[s];
    const uint4* row = reinterpret_cast<const uint4*>(b.slab + (size_t)s * SLAB);
    const uint4 r0 = row[0], r1 = row[1];
    uint32_t e[SLAB] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w};
    const uint32_t h = state_pos(w0);
    const bool open = state_partner(w0) == PENDING;
    uint32_t first = open ? NONE : state_partner(w0);
    if (d <= SLAB) {
#pragma unroll
      for (uint32_t k = 0; k < SLAB; ++k) {
        if (k >= d) e[k] = NONE;
        if (open && k == h) first = e[k];
      }
    } else {
      const uint32_t* list = b.ovf + e[0];  // its end is marked
      if (open) first = list[h];
#pragma unroll
      for (uint32_t k = 1; k < 4; ++k) {
        const uint32_t p = h + k, x = p <= d ? list[p] : NONE;
#pragma unroll
        for (uint32_t m = 0; m < 3; ++m)
          if (p % 3u == m) e[2 + 2 * m] = x, e[3 + 2 * m] = p;
      }
    }
    const unsigned long long w = ev_word(ev_class(state_species(w0)), d > SLAB ? EV_LONG : 0u, h, first);
    words[l] = w;
    rows[2 * l] = make_uint4(e[0], e[1], e[2], e[3]);
    rows[2 * l + 1] = make_uint4(e[4], e[5], e[6], e[7]);
    // a word that was open: publish an upper endpoint of another pair across blocks (the others are)
    if (open && first != NONE && entry_id(first) - t.lo >= t.n && s > entry_id(first))
      st_relaxed(b.wstate + s, pack_state(first, h, (int)(hi32(w) >> 30)));
  }
  __syncthreads();
  // the first pairs: every lower endpoint queues its own; crossing vertices to the watchers
  const uint32_t upto = (t.n + 31u) & ~31u;
  for (uint32_t l = threadIdx.x; l < upto; l += EV_THREADS) {  // whole warps
    const bool live = l < t.n;
    const unsigned long long w = live ? words[l] : (unsigned long long)NONE;
    const uint32_t y = entry_id((uint32_t)w) - t.lo;
    const bool end = (uint32_t)w == NONE, in = !end && y < t.n;
    const bool ready = in && l < y && entry_id((uint32_t)words[y]) == t.lo + l;
    ev_push(t, __ballot_sync(0xffffffffu, ready), l, __ballot_sync(0xffffffffu, live && !end && !in), l,
            __popc(__ballot_sync(0xffffffffu, live && end)));
    if (ready) reinterpret_cast<uint32_t*>(words + l)[1] |= EV_CLAIM;  // (the entry, all that others read here, stays)
  }
  __syncthreads();
  if (threadIdx.x < EV_WATCHERS * 32)
    ev_watch(b, t, ctrl, t0);
  else
    ev_work(b, t, ctrl, t0);
  __syncthreads();
  // every owned list is done: the words hold the final species, written back once per vertex that had
  // pairs (values outside 1..3 are as they were)
  for (uint32_t l = threadIdx.x; l < t.n; l += EV_THREADS) {
    const uint32_t state = hi32(words[l]);
    if ((state & EV_POS) && state >> 30) b.species[b.sid[t.lo + l]] = (int8_t)(state >> 30);
  }
}

// The groups of the rule (ev_taken: k_rounds leaves them out), when the ensembles fit the blocks; else nothing.
__global__ void __launch_bounds__(EV_THREADS, 2) k_rounds_events(Bufs b, StepArgs a, Ctrl* ctrl) {
  __shared__ uint32_t cw[2];
  __shared__ TileGroups tg;
  extern __shared__ unsigned long long ev_raw[];
  if (threadIdx.x == 0) {
    // where fewer than half of the entries are in long lists no group is worth the look (15 us at 7 neighbours)
    const unsigned long long in_long = ((volatile unsigned long long*)&ctrl->ovf_used)[0];
    cw[0] = ((volatile uint32_t*)&ctrl->halt)[0] || 2 * in_long < ((volatile unsigned long long*)&ctrl->n_dir)[0];
    cw[1] = ((volatile uint32_t*)&ctrl->n_valid)[0];
  }
  __syncthreads();
  if (cw[0] || cw[1] == 0u) return;
  if (b.plog || a.test_wait_ns) return;  // logged steps and the injected failure are k_rounds' own
  make_groups(b, cw[1], gridDim.x * EV_VMAX, reinterpret_cast<uint32_t*>(ev_raw), (uint32_t)(EV_SMEM / sizeof(uint32_t)), tg, true);
  if (tg.n <= 0 || !tg.taken) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) ctrl->ev_taken = 1u;
  const unsigned long long t0 = globaltimer();
  for (int g = 0; g < tg.n; ++g) {
    if (!((tg.taken >> g) & 1ull)) continue;
    ev_group(b, ctrl, t0, tg.lo[g], tg.lo[g + 1]);
    __syncthreads();  // the shared memory is the next group's
  }
}

// Grid of the cooperative launch (0: the kernel does not fit the device).
int events_grid(int device) {
  int sms = 0, per_sm = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  cudaFuncSetAttribute(k_rounds_events, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)EV_SMEM);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_rounds_events, EV_THREADS, EV_SMEM);
  return sms * per_sm;
}

cudaError_t launch_events(const Bufs& b, const StepArgs& a, Ctrl* ctrl, int grid, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(EV_THREADS);
  cfg.dynamicSmemBytes = EV_SMEM;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_rounds_events, b, a, ctrl);
}

}  // namespace lm
