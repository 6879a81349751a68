// Pairwise great-circle distance histogram (lm_distance_histogram, lm_species_histogram,
// include/lm_api.h).
//
// The reference's sandbox computes, for the microbes of one species, the distance of every
// unordered pair with its float32 haversine formula and counts it in a log bin
// (sandbox/pairwise_distance_histogram_distributed.jl:35-46 haversine_distance32, :56-66 the
// per-point loop and the bin round(10 log10(max(1, d))), :68-76 the sum over points, :133-147 one
// histogram per species; sandbox/pairwise_distance_histogram_gpu.jl:14-43 a CUDA tiling of the
// same pairs whose histogram update was left unwritten).
//
// A bin is 26 % wide in distance, so most pairs of two small groups of points share one bin. The
// points of every segment (species) are sorted along a Hilbert curve, and the pairs are counted by
// groups of neighbouring points instead of one by one:
//
//   * work items are the tiles (I, J), I <= J, of 256 x 256 sorted points of a segment; a block loads
//     both tiles (latitude, longitude, cos(latitude), index) and the boxes of their 8-point leaves
//     into shared memory (few of them are shared out by groups of J);
//   * the haversine a = sin^2(dlat / 2) + cos cos sin^2(dlon / 2) of a pair of boxes is bounded from
//     the extremes of dlat, dlon and cos(latitude), first for the 8 x 8 pairs of 32-point groups,
//     then for the leaf pairs of the groups that are left. If every a of a pair of groups lies inside
//     one bin, its pairs are counted at once;
//   * a leaf pair whose bounds straddle one bin boundary is evaluated by two lanes: 64 values of a (as
//     the squared chord of unit vectors) against that boundary's threshold in a;
//   * what is left (close, ragged and diagonal leaf pairs, and those within 0.9 degrees of a pole) is
//     evaluated pair by pair (dh_pair_bin).
//
// The definition of a pair's bin stays the reference's float32 chain (dh_bin: haversine_distance32
// operation by operation, divisions and products rounded as written, the lower index first, with
// CUDA's sinpif / cospif / asinf / log10f; round half to even; bins at or past `bins` go to an
// overflow count, where the reference indexes past its array). The chain's 10 log10 d is off the
// true value by 1.6e-5 at most (log10f within 2 ulp of values up to 7.3, the product by ten rounded
// once, asinf within 2 ulp, the rest below 2e-6), a bound of a taken from the chain's own cosines by
// less than 3e-6, a squared chord by less than 1.8e-5 (dh_two_bins), and the hardware log2 by 1.4e-5
// more. The chain's cosine comes from latitude / 180 rounded to float32, 1.5e-8 at most up to 90 degrees,
// so it is off by 4.7e-8 / cos relative; the unit vectors do not carry that, and the chord differs from
// the chain by 2.1e-7 / cos for it: 1.4e-5 at cos >= DH_COS_VEC = 1/64, below which (and past 90 degrees)
// chords are not taken. So a route decides a pair only when its value lies farther than DH_MARGIN_A =
// 5e-5 (a alone) or DH_MARGIN = 1e-4 (log2) from the boundary; the chain itself decides every other
// pair. LM_HIST_EXACT=1 in the environment makes every pair take the chain (the tests compare the two).
//
// Bound by instruction issue. At 490k microbes on 5 x 5 degrees (three species, 4.0e10 pairs) a call
// took 100.0 ms with every pair evaluated by itself; counted by groups it takes 8.1 ms: 19 % of the
// pairs are compared with a threshold (3.9 ms) and 1 % take the logarithm (0.8 ms).
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <new>
#include <vector>

#include "lm_api.h"
#include "lm_internal.h"

namespace lm {
namespace {

constexpr int DH_THREADS = 128;                // threads per block
constexpr int DH_WARPS = DH_THREADS / 32;
constexpr uint32_t DH_TILE = 256;              // points per tile
constexpr uint32_t DH_GROUP = 32, DH_LEAF = 8; // points per group and per leaf of a tile
constexpr uint32_t DH_GROUPS = DH_TILE / DH_GROUP, DH_LEAVES = DH_TILE / DH_LEAF;
constexpr int DH_COPIES = 4;                   // histogram copies per warp (lanes l and l + 4 share one)
constexpr int DH_BINS_MAX = 256;
constexpr uint32_t DH_FLUSH = 16384;           // items between flushes: at most 2^16 counts each, < 2^32 a word
constexpr int DH_CURVE_BITS = 20;              // 10 a coordinate: two digits of the radix sort

struct DhSeg {
  unsigned long long item0;  // first work item of the segment
  uint32_t start, pstart, n; // first point in sorted order and in the padded point arrays, points
  uint32_t tile0;            // first tile
};

// The unit vector of a tile's first point; the tile's points are kept relative to it.
struct DhTile {
  double x, y, z;
  float radius;  // distance of its farthest point
};

// Control words of one call.
struct DhCtl {
  unsigned long long n_items;  // work items of all segments
  unsigned long long next;     // next item to hand out
  uint32_t box[4];             // ordered-int encoded min latitude, min longitude, max latitude, max longitude
  uint32_t bad;                // a point of a segment is not finite
  uint32_t count[3];           // points per species
};

// Box of the points of a leaf or a group: extremes of latitude, longitude and cos(latitude).
struct DhBox {
  float la0, la1, lo0, lo1, c0, c1;
};

__device__ __forceinline__ DhBox dh_join(const DhBox& a, const DhBox& b) {
  return DhBox{fminf(a.la0, b.la0), fmaxf(a.la1, b.la1), fminf(a.lo0, b.lo0),
               fmaxf(a.lo1, b.lo1), fminf(a.c0, b.c0),   fmaxf(a.c1, b.c1)};
}

// Segment of point i: its species (1..3 -> 0..2, other values are in no segment) or the segment whose
// range holds it.
__device__ __forceinline__ uint32_t dh_segment(uint32_t i, const int8_t* __restrict__ species,
                                               const DhSeg* __restrict__ segs, uint32_t n_seg) {
  if (species) {
    const int k = species[i];
    return k >= 1 && k <= 3 ? (uint32_t)(k - 1) : n_seg;
  }
  uint32_t lo = 0, hi = n_seg;  // the last segment starting at or before i (empty ones share a start)
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) / 2;
    if (segs[mid].start <= i) lo = mid; else hi = mid;
  }
  return lo;
}

// Extremes of the coordinates, the non-finite flag and the points per species.
__global__ void __launch_bounds__(256) k_dh_box(const float* __restrict__ lat, const float* __restrict__ lon,
                                                const int8_t* __restrict__ species, uint32_t n,
                                                DhCtl* __restrict__ ctl) {
  const uint32_t lane = threadIdx.x & 31u;
  float b[4] = {INFINITY, INFINITY, INFINITY, INFINITY};  // min lat, min lon, min -lat, min -lon
  bool bad = false;
  uint32_t cnt[3] = {0, 0, 0};
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    if (species) {
      const int k = species[i];
      if (k < 1 || k > 3) continue;
#pragma unroll
      for (int q = 0; q < 3; ++q) cnt[q] += k == q + 1 ? 1u : 0u;
    }
    const float a = lat[i], o = lon[i];
    bad |= !(isfinite(a) && isfinite(o));
    b[0] = fminf(b[0], a);
    b[1] = fminf(b[1], o);
    b[2] = fminf(b[2], -a);
    b[3] = fminf(b[3], -o);
  }
#pragma unroll
  for (int q = 0; q < 4; ++q)
    for (int o = 16; o > 0; o >>= 1) b[q] = fminf(b[q], __shfl_xor_sync(0xffffffffu, b[q], o));
#pragma unroll
  for (int q = 0; q < 3; ++q)
    for (int o = 16; o > 0; o >>= 1) cnt[q] += __shfl_xor_sync(0xffffffffu, cnt[q], o);
  bad = __any_sync(0xffffffffu, bad);
  if (lane != 0) return;
  if (bad) ctl->bad = 1u;
  if (b[0] <= -b[2]) {
    atomicMin(&ctl->box[0], enc_f(b[0]));
    atomicMin(&ctl->box[1], enc_f(b[1]));
    atomicMax(&ctl->box[2], enc_f(-b[2]));
    atomicMax(&ctl->box[3], enc_f(-b[3]));
  }
#pragma unroll
  for (int q = 0; q < 3; ++q)
    if (cnt[q]) atomicAdd(&ctl->count[q], cnt[q]);
}

// Work items of a segment of n points: the tile pairs I <= J.
__host__ __device__ inline unsigned long long dh_items(uint32_t n) {
  const unsigned long long t = ((unsigned long long)n + DH_TILE - 1) / DH_TILE;
  return t * (t + 1) / 2;
}
__host__ __device__ inline uint32_t dh_tiles(uint32_t n) { return (n + DH_TILE - 1) / DH_TILE; }
__host__ __device__ inline uint32_t dh_padded(uint32_t n) { return (n + DH_LEAF - 1) / DH_LEAF * DH_LEAF; }

// The three species' segments from their counts.
__global__ void k_dh_species_segs(DhCtl* ctl, DhSeg* segs) {
  unsigned long long items = 0;
  uint32_t start = 0, pstart = 0, tiles = 0;
  for (int q = 0; q < 3; ++q) {
    const uint32_t m = ctl->count[q];
    segs[q] = DhSeg{items, start, pstart, m, tiles};
    items += dh_items(m);
    tiles += dh_tiles(m);
    start += m;
    pstart += dh_padded(m);
  }
  ctl->n_items = items;
}

// Sort key: segment, then the point's place along Hilbert's curve over the common bounding box (mb
// bits). Any order of the points gives the same counts; this one makes the leaves small (8 points of a
// lattice's species span 0.032 degrees on average, 0.055 in Morton order).
__global__ void __launch_bounds__(256) k_dh_key(const float* __restrict__ lat, const float* __restrict__ lon,
                                                const int8_t* __restrict__ species, uint32_t n,
                                                const DhSeg* __restrict__ segs, uint32_t n_seg, int mb,
                                                const DhCtl* __restrict__ ctl, uint32_t* __restrict__ key) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t s = dh_segment(i, species, segs, n_seg);
  uint32_t m = 0;
  if (mb > 0 && s < n_seg) {
    const float a0 = dec_f(ctl->box[0]), o0 = dec_f(ctl->box[1]);
    const float cells = (float)(1u << (mb / 2));
    const float wa = dec_f(ctl->box[2]) - a0, wo = dec_f(ctl->box[3]) - o0;
    // a zero extent or an overflowing one gives NaN or 0 here, which the clamp takes to cell 0
    const uint32_t qa = (uint32_t)fminf(fmaxf((lat[i] - a0) / wa * cells, 0.f), cells - 1.f);
    const uint32_t qo = (uint32_t)fminf(fmaxf((lon[i] - o0) / wo * cells, 0.f), cells - 1.f);
    m = hilbert_place(qa, qo, mb / 2);
  }
  key[i] = (s << mb) | m;
}

// One block per tile: its sorted points into the padded arrays (every segment starts on a leaf) as
// (latitude, longitude, cos(latitude), index in the caller's order) and as the unit vector relative to
// the tile's first point, taken in float64 and rounded once.
__global__ void __launch_bounds__(DH_TILE) k_dh_gather(const float* __restrict__ lat, const float* __restrict__ lon,
                                                       const uint32_t* __restrict__ sval,
                                                       const DhSeg* __restrict__ segs, uint32_t n_seg,
                                                       float4* __restrict__ pts, float4* __restrict__ vec,
                                                       DhTile* __restrict__ tiles) {
  __shared__ double first[3];
  __shared__ float red[DH_TILE / 32];
  uint32_t lo = 0, hi = n_seg;  // the last segment whose tiles start at or before this one
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) / 2;
    if (segs[mid].tile0 <= blockIdx.x) lo = mid; else hi = mid;
  }
  const DhSeg S = segs[lo];
  const uint32_t k = (blockIdx.x - S.tile0) * DH_TILE + threadIdx.x;
  if (blockIdx.x - S.tile0 >= dh_tiles(S.n)) return;  // block-uniform: past the last tile
  double v[3] = {0.0, 0.0, 0.0};
  if (k < S.n) {
    const uint32_t i = sval[S.start + k];
    const float a = lat[i], o = lon[i];
    pts[S.pstart + k] = make_float4(a, o, cospif(__fdiv_rn(a, 180.0f)), __uint_as_float(i));
    double sa, ca, so, co;
    sincospi((double)a / 180.0, &sa, &ca);
    sincospi((double)o / 180.0, &so, &co);
    v[0] = ca * co;
    v[1] = ca * so;
    v[2] = sa;
  }
  if (threadIdx.x == 0) first[0] = v[0], first[1] = v[1], first[2] = v[2];
  __syncthreads();
  float r2 = 0.f;
  if (k < S.n) {
    const float x = (float)(v[0] - first[0]), y = (float)(v[1] - first[1]), z = (float)(v[2] - first[2]);
    vec[S.pstart + k] = make_float4(x, y, z, 0.f);
    r2 = fmaf(x, x, fmaf(y, y, z * z));
  }
  for (int o = 16; o > 0; o >>= 1) r2 = fmaxf(r2, __shfl_xor_sync(0xffffffffu, r2, o));
  if ((threadIdx.x & 31u) == 0) red[threadIdx.x / 32] = r2;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (uint32_t w = 1; w < DH_TILE / 32; ++w) r2 = fmaxf(r2, red[w]);
    tiles[blockIdx.x] = DhTile{v[0], v[1], v[2], sqrtf(r2)};
  }
}

// haversine_distance32 (lat, lon in degrees, c = cospi(lat / 180)), then the bin.
__device__ __forceinline__ int dh_bin(float la1, float lo1, float c1, float la2, float lo2, float c2, float R) {
  const float dlat = __fsub_rn(la2, la1), dlon = __fsub_rn(lo2, lo1);
  const float d1 = sinpif(__fdiv_rn(dlat, 360.0f));
  const float d2 = sinpif(__fdiv_rn(dlon, 360.0f));
  const float t = __fmul_rn(__fmul_rn(__fmul_rn(d2, d2), c1), c2);
  const float a = __fadd_rn(__fmul_rn(d1, d1), t);
  const float c = __fmul_rn(2.0f, asinf(fminf(1.0f, __fsqrt_rn(a))));
  const float d = __fmul_rn(R, c);
  return (int)rintf(__fmul_rn(10.0f, log10f(fmaxf(1.0f, d))));
}

constexpr float DH_MARGIN = 1e-4f;      // routes through the hardware log2
constexpr float DH_MARGIN_A = 5e-5f;    // routes that compare a with a threshold
constexpr float DH_COS_VEC = 0.015625f;  // smallest cos(latitude) of the leaf pairs decided by chords
constexpr float DH_PI_360 = 8.72664625997164788e-3f;  // pi / 360
constexpr float DH_NEAR_DEG = 24.0f;  // |dlat|, |dlon| up to which dh_hav<true> holds

// sin x for |x| <= pi / 2: Taylor series to x^11 (truncation below 6e-8 relative there).
__device__ __forceinline__ float dh_sin(float x) {
  const float z = x * x;
  float p = -2.50521083854417188e-8f;  // -1 / 11!
  p = fmaf(p, z, 2.75573192239858907e-6f);  // 1 / 9!
  p = fmaf(p, z, -1.98412698412698413e-4f);  // -1 / 7!
  p = fmaf(p, z, 8.33333333333333333e-3f);   // 1 / 5!
  p = fmaf(p, z, -1.66666666666666667e-1f);  // -1 / 3!
  return fmaf(x * z, p, x);
}

// a / (pi / 360)^2 for NEAR, else a itself: the haversine of a pair from dlat, dlon (degrees) and
// cc = c1 c2. NEAR (|dlat|, |dlon| <= 24 degrees, x = half the difference <= 0.21): sin^2 x =
// z - z^2 / 3 + 2 z^3 / 45 - z^4 / 315 with z = x^2 (truncation below 1e-9 relative), the scale of
// z folded into the coefficients. Otherwise |dlat|, |dlon| <= 180.
template <bool NEAR>
__device__ __forceinline__ float dh_hav(float dlat, float dlon, float cc) {
  if (NEAR) {
    constexpr float k = DH_PI_360 * DH_PI_360;
    constexpr float p1 = -k / 3.0f, p2 = k * k * 2.0f / 45.0f, p3 = -k * k * k / 315.0f;
    const float za = dlat * dlat, zo = dlon * dlon;
    const float pa = fmaf(fmaf(fmaf(p3, za, p2), za, p1), za, 1.0f);
    const float po = fmaf(fmaf(fmaf(p3, zo, p2), zo, p1), zo, 1.0f);
    return fmaf(za, pa, zo * po * cc);
  }
  const float d1 = dh_sin(dlat * DH_PI_360), d2 = dh_sin(dlon * DH_PI_360);
  return fmaf(d1, d1, d2 * d2 * cc);
}
template <bool NEAR>
__device__ __forceinline__ float dh_hav_scale() { return NEAR ? DH_PI_360 * DH_PI_360 : 1.0f; }

// Everything of a call that the pair routes need.
struct DhRule {
  const float2* thr;  // [bins] boundary k between bins k and k + 1, as values of a: below .x the chain's
                      // bin is at most k, above .y at least k + 1
  float a_min;        // a of d = 1.5 m: the routes on a hold from here ...
  float R, log_2R10;  // 10 log10(2 R)
  int bins, exact;
};
constexpr float DH_A_MAX = 0.9f;  // ... to here (near the antipode 10 log10 d is too steep in a)

// The chain on a pair, the lower index first (it is not symmetric in float32).
__device__ __forceinline__ int dh_chain(const float4& p, const float4& q, float R) {
  const bool in_order = __float_as_uint(p.w) < __float_as_uint(q.w);
  const float4 &u = in_order ? p : q, &v = in_order ? q : p;
  return dh_bin(u.x, u.y, u.z, v.x, v.y, v.z, R);
}

// 10 log10 d for 0 < a <= 1/16: 10 log10(2 R) + 5 log10 a + 10 log10(asin(s) / s), s = sqrt(a), with
// ln(asin(s) / s) = a / 6 + 11 a^2 / 180 + 191 a^3 / 5670 + ... (truncation below 2e-6 in 10 log10 d).
constexpr float DH_A_SERIES = 0.0625f;
__device__ __forceinline__ float dh_db(float a, const DhRule& r) {
  float t = fmaf(a, 0.146297f, 0.265402f);  // 191 / 5670 and 11 / 180 times 10 / ln 10
  t = fmaf(a, t, 0.723824f);                // 10 / (6 ln 10)
  return fmaf(1.50514997831990598f, __log2f(a), fmaf(a, t, r.log_2R10));  // 5 log10(2)
}

// Bin of one pair: the series where it holds (1.5 m <= d, a <= 1/16), else the chain.
template <bool NEAR>
__device__ __forceinline__ int dh_pair_bin(const float4& p, const float4& q, const DhRule& r) {
  const float dlat = q.x - p.x, dlon = q.y - p.y;
  const float a = dh_hav<NEAR>(dlat, dlon, p.z * q.z) * dh_hav_scale<NEAR>();
  const float x = dh_db(a, r);
  const float k = rintf(x);
  const bool in_range = NEAR || (fabsf(dlat) <= 180.0f && fabsf(dlon) <= 180.0f);
  if (!r.exact && in_range && a >= r.a_min && a <= DH_A_SERIES && fabsf(x - k) < 0.5f - DH_MARGIN)
    return min((int)k, r.bins);
  return min(dh_chain(p, q, r.R), r.bins);
}

// What the boxes u, v say of their pairs: lo and hi bound every a (lo > hi: the routes on a do not
// hold for them).
template <bool NEAR>
__device__ __forceinline__ void dh_bounds(const DhBox& u, const DhBox& v, const DhRule& r, float* lo, float* hi) {
  const float a0 = fmaxf(0.f, fmaxf(v.la0 - u.la1, u.la0 - v.la1)), a1 = fmaxf(v.la1 - u.la0, u.la1 - v.la0);
  const float o0 = fmaxf(0.f, fmaxf(v.lo0 - u.lo1, u.lo0 - v.lo1)), o1 = fmaxf(v.lo1 - u.lo0, u.lo1 - v.lo0);
  const bool ok = (NEAR || (a1 <= 180.f && o1 <= 180.f)) && u.c0 >= 0.f && v.c0 >= 0.f && !r.exact;
  *lo = dh_hav<NEAR>(a0, o0, u.c0 * v.c0) * dh_hav_scale<NEAR>();
  *hi = dh_hav<NEAR>(a1, o1, u.c1 * v.c1) * dh_hav_scale<NEAR>();
  if (!(ok && *lo >= r.a_min && *hi <= DH_A_MAX)) {
    *lo = 1.f;
    *hi = 0.f;
  }
}

// Are all |dlat| and |dlon| of the boxes' pairs at most DH_NEAR_DEG?
__device__ __forceinline__ bool dh_near(const DhBox& u, const DhBox& v) {
  return fmaxf(fmaxf(v.la1 - u.la0, u.la1 - v.la0), fmaxf(v.lo1 - u.lo0, u.lo1 - v.lo0)) <= DH_NEAR_DEG;
}

// First boundary that lies above a (bins when none does): a is in that bin or, within the margin of
// the boundary below, in the one below.
__device__ __forceinline__ int dh_first_above(float a, const DhRule& r, const float2* thr) {
  // the guess ignores asin(s) / s, which adds at most 2 bins
  int k = (int)rintf(fmaf(1.50514997831990598f, __log2f(a), r.log_2R10));
  k = min(max(k, 0), r.bins);
  while (k < r.bins && a >= thr[k].x) ++k;
  while (k > 0 && a < thr[k - 1].x) --k;
  return k;
}

// Bins of the bounds: the pairs lie in bin *k (return 1), in bins *k and *k + 1 (2) or in more (0).
__device__ __forceinline__ int dh_span(float lo, float hi, const DhRule& r, const float2* thr, int* k) {
  if (lo > hi) return 0;
  if (hi <= DH_A_SERIES) {
    const int k0 = max((int)floorf(dh_db(lo, r) + (0.5f - DH_MARGIN)), 0);
    const int k1 = (int)floorf(dh_db(hi, r) + (0.5f + DH_MARGIN));
    *k = min(k0, r.bins);
    return min(k1, r.bins) - *k <= 1 ? min(k1, r.bins) - *k + 1 : 0;
  }
  const int ka = dh_first_above(lo, r, thr);
  const int kb = ka < r.bins && hi >= thr[ka].x ? dh_first_above(hi, r, thr) : ka;
  // lo above boundary ka - 1 by the margin, else that boundary is open too
  const int k0 = ka > 0 && lo <= thr[ka - 1].y ? ka - 1 : ka;
  *k = k0;
  return kb - k0 <= 1 ? kb - k0 + 1 : 0;
}

__device__ void dh_flush(uint32_t* hist, int nb, unsigned long long* out) {
  __syncthreads();
  for (int b = threadIdx.x; b < nb; b += DH_THREADS) {
    unsigned long long s = 0;
    for (int w = 0; w < DH_WARPS; ++w)
      for (int q = 0; q < DH_COPIES; ++q) {
        uint32_t* p = hist + ((size_t)w * nb + b) * DH_COPIES + q;
        s += *p;
        *p = 0;
      }
    if (s) atomicAdd(out + b, s);
  }
  __syncthreads();
}

constexpr uint32_t DH_UNSURE = 128;
struct DhShared {
  float4 pt[2][DH_TILE];          // the points of tiles I and J
  float4 vec[2][DH_TILE];         // and their unit vectors, relative to the tile's first point
  DhBox leaf[2][DH_LEAVES];       // boxes of their leaves
  uint32_t open[DH_GROUPS * DH_GROUPS];     // group pairs left to their leaves
  uint32_t list[DH_LEAVES * DH_LEAVES];     // leaf pairs left: two-bin ones from the front, others from the back
  uint32_t unsure[DH_UNSURE];     // rows of 8 pairs with one too near its boundary: point of I, leaf of J, boundary
  uint32_t n_open, n_two, n_gen, n_unsure, wide;
  float dx, dy, dz;               // first point of tile J minus first point of tile I
  float a_vec;                    // a from which the vectors serve (dh_two_bins)
  unsigned long long next;
};

// How a chord's square c (4 a) falls between the thresholds of a boundary: 1 below, 0 above, a fraction
// within the margin.
struct DhStep {
  float s, t;
  __device__ DhStep(float2 thr) : s(-0.25f / (thr.y - thr.x)), t(thr.y / (thr.y - thr.x)) {}
  __device__ __forceinline__ float operator()(float c) const { return __saturatef(fmaf(c, s, t)); }
};

// The leaf pairs of the list that straddle one boundary, by two lanes each: the 8 points of J in
// registers against 4 points of I. a is a quarter of the squared chord of the unit vectors, kept
// relative to a point of each tile, so a coordinate difference is off by at most 4 roundings of the
// tiles' extent E; leaf pairs closer than E / 8 are not listed here (a_vec), so a is off by less
// than 8e-6 relative. The lanes start their leaves at different points, so the 16-byte loads of a
// quarter warp fall into different banks. A row of 8 pairs with one within the margin of the boundary
// (the sum of f differs from the sum of f^2) is left for dh_unsure, or settled here when its queue is
// full.
__device__ __forceinline__ float dh_chord2(const float4& p, float x, float y, float z) {
  const float dx = p.x - x, dy = p.y - y, dz = p.z - z;
  return fmaf(dx, dx, fmaf(dy, dy, dz * dz));
}

__device__ __forceinline__ void dh_settle(const DhShared& sh, uint32_t sj, uint32_t i, uint32_t j, uint32_t k,
                                          const DhRule& r, const float2* thr, uint32_t* mine) {
  const float4 q = sh.vec[sj][j];
  const float f = DhStep(thr[k])(dh_chord2(sh.vec[0][i], q.x + sh.dx, q.y + sh.dy, q.z + sh.dz));
  const int b = f == 1.f ? (int)k : f == 0.f ? (int)k + 1 : min(dh_chain(sh.pt[0][i], sh.pt[sj][j], r.R), r.bins);
  atomicAdd(mine + b * DH_COPIES, 1u);
}

__device__ __forceinline__ void dh_two_bins(DhShared& sh, uint32_t sj, const DhRule& r, const float2* thr,
                                            uint32_t* mine) {
  const uint32_t lane = threadIdx.x & 7u;
  for (uint32_t e = threadIdx.x; e < 2 * sh.n_two; e += DH_THREADS) {
    const uint32_t code = sh.list[e / 2], li = code & 31u, lj = (code >> 5) & 31u, k = code >> 10;
    const DhStep step(thr[k]);
    float x[DH_LEAF], y[DH_LEAF], z[DH_LEAF];
#pragma unroll
    for (uint32_t t = 0; t < DH_LEAF; ++t) {
      const float4 q = sh.vec[sj][lj * DH_LEAF + ((t + lane) & 7u)];
      x[t] = q.x + sh.dx;
      y[t] = q.y + sh.dy;
      z[t] = q.z + sh.dz;
    }
    float below = 0.f;
    uint32_t rows = 0;
#pragma unroll 2
    for (uint32_t t = 0; t < DH_LEAF / 2; ++t) {
      // the entry's two lanes share lane / 2, so their rows differ by 4
      const uint32_t i = li * DH_LEAF + ((t + (e & 1u) * (DH_LEAF / 2) + lane / 2) & 7u);
      const float4 p = sh.vec[0][i];
      float b = 0.f, b2 = 0.f;
#pragma unroll
      for (uint32_t u = 0; u < DH_LEAF; ++u) {
        const float f = step(dh_chord2(p, x[u], y[u], z[u]));
        b += f;
        b2 = fmaf(f, f, b2);
      }
      if (b == b2) {
        below += b;
        ++rows;
      } else {
        const uint32_t at = atomicAdd(&sh.n_unsure, 1u);
        if (at < DH_UNSURE) {
          sh.unsure[at] = i | (lj << 8) | (k << 13);
        } else {
#pragma unroll 1
          for (uint32_t u = 0; u < DH_LEAF; ++u) dh_settle(sh, sj, i, lj * DH_LEAF + u, k, r, thr, mine);
        }
      }
    }
    const uint32_t m = __float2uint_rn(below);  // (a place just below 1 may leave the sum an ulp short)
    if (m) atomicAdd(mine + k * DH_COPIES, m);
    if (m != rows * DH_LEAF) atomicAdd(mine + (k + 1) * DH_COPIES, rows * DH_LEAF - m);
  }
}

// The pairs of the queued rows, one lane per pair.
__device__ __forceinline__ void dh_unsure(const DhShared& sh, uint32_t sj, const DhRule& r, const float2* thr,
                                          uint32_t* mine) {
  const uint32_t n = min(sh.n_unsure, DH_UNSURE) * DH_LEAF;
  for (uint32_t w = threadIdx.x; w < n; w += DH_THREADS) {
    const uint32_t code = sh.unsure[w / DH_LEAF];
    dh_settle(sh, sj, code & 255u, ((code >> 8) & 31u) * DH_LEAF + (w & 7u), code >> 13, r, thr, mine);
  }
}

// The other leaf pairs, pair by pair: four lanes per leaf pair, two points of I each.
template <bool NEAR>
__device__ __forceinline__ void dh_general(const DhShared& sh, uint32_t sj, bool diagonal, uint32_t ni, uint32_t nj,
                                           const DhRule& r, uint32_t* mine) {
  const uint32_t n = 4u * sh.n_gen;
  for (uint32_t w = threadIdx.x; w < n; w += DH_THREADS) {
    const uint32_t code = sh.list[DH_LEAVES * DH_LEAVES - 1u - w / 4u], li = code & 31u, lj = (code >> 5) & 31u;
    const uint32_t i0 = li * DH_LEAF, j0 = lj * DH_LEAF;
    const uint32_t mi = min(DH_LEAF, ni - i0), mj = min(DH_LEAF, nj - j0);
    for (uint32_t t = w & 3u; t < mi; t += 4) {
      const float4 p = sh.pt[0][i0 + t];
      for (uint32_t u = diagonal && li == lj ? t + 1 : 0u; u < mj; ++u)
        atomicAdd(mine + dh_pair_bin<NEAR>(p, sh.pt[sj][j0 + u], r) * DH_COPIES, 1u);
    }
  }
}

// The leaf pairs of the open group pairs: counted at once, or listed.
template <bool NEAR>
__device__ __forceinline__ void dh_leaf_pairs(DhShared& sh, uint32_t sj, bool diagonal, uint32_t ni, uint32_t nj,
                                              const DhRule& r, const float2* thr, uint32_t* mine) {
  const uint32_t lvi = (ni + DH_LEAF - 1) / DH_LEAF, lvj = (nj + DH_LEAF - 1) / DH_LEAF;
  const uint32_t n = sh.n_open * 16u;
  for (uint32_t t = threadIdx.x; t < n; t += DH_THREADS) {
    const uint32_t o = sh.open[t / 16u];
    const uint32_t a = 4u * (o & 15u) + (t & 3u), b = 4u * (o >> 4) + ((t >> 2) & 3u);
    if (a >= lvi || b >= lvj || (diagonal && a > b)) continue;
    const uint32_t ma = min(DH_LEAF, ni - a * DH_LEAF), mb = min(DH_LEAF, nj - b * DH_LEAF);
    int k = 0, span = 0;
    float lo = 0.f, hi;
    if (!(diagonal && a == b)) {
      dh_bounds<NEAR>(sh.leaf[0][a], sh.leaf[sj][b], r, &lo, &hi);
      span = dh_span(lo, hi, r, thr, &k);
    }
    if (span == 1)
      atomicAdd(mine + k * DH_COPIES, ma * mb);
    else if (span == 2 && ma * mb == DH_LEAF * DH_LEAF && lo >= sh.a_vec &&
             fminf(sh.leaf[0][a].c0, sh.leaf[sj][b].c0) >= DH_COS_VEC)
      sh.list[atomicAdd(&sh.n_two, 1u)] = a | (b << 5) | ((uint32_t)k << 10);
    else
      sh.list[DH_LEAVES * DH_LEAVES - 1u - atomicAdd(&sh.n_gen, 1u)] = a | (b << 5);
  }
}

__device__ __forceinline__ DhBox dh_group_box(const DhBox* leaf, uint32_t g, uint32_t n_leaves) {
  DhBox b = leaf[4 * g];
  for (uint32_t k = 4 * g + 1; k < min(4 * g + 4, n_leaves); ++k) b = dh_join(b, leaf[k]);
  return b;
}

// Points of a tile (n of them from pts and vec) and the boxes of its leaves.
__device__ __forceinline__ void dh_load_tile(const float4* __restrict__ pts, const float4* __restrict__ vecs, uint32_t n,
                                             float4* pt, float4* vec, DhBox* leaf) {
  for (uint32_t t = threadIdx.x; t < DH_TILE; t += DH_THREADS) {
    DhBox b{INFINITY, -INFINITY, INFINITY, -INFINITY, INFINITY, -INFINITY};
    if (t < n) {
      const float4 p = pts[t];
      vec[t] = vecs[t];
      pt[t] = p;
      // past 90 degrees (where latitude / 180 may round to anything) no box serves: as for a negative cosine
      b = DhBox{p.x, p.x, p.y, p.y, fabsf(p.x) <= 90.f ? p.z : -1.f, p.z};
    }
    for (int o = 4; o > 0; o >>= 1) {
      const DhBox c{__shfl_xor_sync(0xffffffffu, b.la0, o), __shfl_xor_sync(0xffffffffu, b.la1, o),
                    __shfl_xor_sync(0xffffffffu, b.lo0, o), __shfl_xor_sync(0xffffffffu, b.lo1, o),
                    __shfl_xor_sync(0xffffffffu, b.c0, o),  __shfl_xor_sync(0xffffffffu, b.c1, o)};
      b = dh_join(b, c);
    }
    if ((t & (DH_LEAF - 1)) == 0) leaf[t / DH_LEAF] = b;
  }
}

// SHARED_OUT: fewer items than blocks are shared out by parts, the groups of tile J in turn, so that all blocks have
// work (one form for both took 0.5 % more at 490,000).
template <bool SHARED_OUT>
__global__ void __launch_bounds__(DH_THREADS, 8) k_dist_hist(const float4* __restrict__ pts,
                                                          const float4* __restrict__ vec,
                                                          const DhTile* __restrict__ tiles,
                                                          const DhSeg* __restrict__ segs, uint32_t n_seg,
                                                          DhCtl* __restrict__ ctl, DhRule rule,
                                                          unsigned long long* __restrict__ counts) {
  __shared__ DhShared sh;
  extern __shared__ uint32_t hist[];  // [warp][bin][copy], bin = bins is the overflow; then the thresholds
  if (ctl->bad) return;
  const int nb = rule.bins + 1;
  float2* thr = reinterpret_cast<float2*>(hist + (size_t)DH_WARPS * nb * DH_COPIES);
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  for (int q = threadIdx.x; q < DH_WARPS * nb * DH_COPIES; q += DH_THREADS) hist[q] = 0;
  for (int q = threadIdx.x; q < rule.bins; q += DH_THREADS) thr[q] = rule.thr[q];
  uint32_t* mine = hist + (size_t)warp * nb * DH_COPIES + (lane & (DH_COPIES - 1));
  uint32_t cut = 0;  // 2^cut parts an item
  while (SHARED_OUT && cut < 3u && (ctl->n_items << (cut + 1u)) <= gridDim.x) ++cut;
  const unsigned long long n_items = ctl->n_items << cut;
  // consecutive items share their tile J; a share small enough that the last blocks do not wait long
  const unsigned long long share = min(8ull, max(1ull, n_items / (8ull * gridDim.x)));
  int cur = -1;
  uint32_t since = 0;
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) sh.next = atomicAdd(&ctl->next, share);
    __syncthreads();
    const unsigned long long w0 = sh.next, w1 = min(n_items, w0 + share);
    if (w0 >= n_items) break;
    unsigned long long J = ~0ull, I = 0;
    bool have_j = false;
    for (unsigned long long w = w0; w < w1; ++w) {
      int sg = cur < 0 ? 0 : cur;  // a block's items come in segment order
      while (sg + 1 < (int)n_seg && (w >> cut) >= segs[sg + 1].item0) ++sg;
      if (sg != cur || since >= DH_FLUSH) {  // block-uniform
        if (cur >= 0) dh_flush(hist, nb, counts + (size_t)cur * nb);
        if (sg != cur) J = ~0ull;
        cur = sg;
        since = 0;
      }
      const DhSeg S = segs[sg];
      if (J == ~0ull) {
        // item t of the segment is tile pair (I, J) with J (J + 1) / 2 <= t < (J + 1) (J + 2) / 2
        const unsigned long long t = (w >> cut) - S.item0;
        J = (unsigned long long)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
        while (J * (J + 1) / 2 > t) --J;
        while ((J + 1) * (J + 2) / 2 <= t) ++J;
        I = t - J * (J + 1) / 2;
        have_j = false;
      } else if ((w & ((1u << cut) - 1u)) == 0u && ++I > J) {
        ++J;
        I = 0;
        have_j = false;
      }
      const uint32_t i0 = (uint32_t)I * DH_TILE, j0 = (uint32_t)J * DH_TILE;
      const uint32_t ni = min(DH_TILE, S.n - i0), nj = min(DH_TILE, S.n - j0);
      const uint32_t gi = (ni + DH_GROUP - 1) / DH_GROUP, gj = (nj + DH_GROUP - 1) / DH_GROUP;
      const uint32_t lvi = (ni + DH_LEAF - 1) / DH_LEAF, lvj = (nj + DH_LEAF - 1) / DH_LEAF;
      const bool diagonal = I == J;
      const uint32_t sj = diagonal ? 0u : 1u;  // where tile J's points are
      __syncthreads();  // the previous tiles are no longer read
      dh_load_tile(pts + S.pstart + i0, vec + S.pstart + i0, ni, sh.pt[0], sh.vec[0], sh.leaf[0]);
      if (!diagonal && !have_j) {
        dh_load_tile(pts + S.pstart + j0, vec + S.pstart + j0, nj, sh.pt[1], sh.vec[1], sh.leaf[1]);
        have_j = true;
      }
      if (threadIdx.x == 0) {
        sh.n_open = sh.n_two = sh.n_gen = sh.n_unsure = sh.wide = 0;
        const DhTile &u = tiles[S.tile0 + (uint32_t)I], &v = tiles[S.tile0 + (uint32_t)J];
        const float dx = (float)(v.x - u.x), dy = (float)(v.y - u.y), dz = (float)(v.z - u.z);
        const float extent = sqrtf(fmaf(dx, dx, fmaf(dy, dy, dz * dz))) + u.radius + v.radius;
        sh.dx = dx;
        sh.dy = dy;
        sh.dz = dz;
        sh.a_vec = extent * extent * (1.0f / 256.0f);  // chord >= extent / 8
      }
      __syncthreads();
      // pairs of 32-point groups
      for (uint32_t g = threadIdx.x; g < gi * gj; g += DH_THREADS) {
        const uint32_t a = g % gi, b = g / gi;
        if ((diagonal && a > b) || ((b ^ (uint32_t)w) & ((1u << cut) - 1u))) continue;
        const DhBox u = dh_group_box(sh.leaf[0], a, lvi), v = dh_group_box(sh.leaf[sj], b, lvj);
        if (!dh_near(u, v)) sh.wide = 1u;
        float lo, hi;
        dh_bounds<false>(u, v, rule, &lo, &hi);
        int k;
        if (!(diagonal && a == b) && dh_span(lo, hi, rule, thr, &k) == 1)
          atomicAdd(mine + k * DH_COPIES, min(DH_GROUP, ni - a * DH_GROUP) * min(DH_GROUP, nj - b * DH_GROUP));
        else
          sh.open[atomicAdd(&sh.n_open, 1u)] = a | (b << 4);
      }
      __syncthreads();
      const bool wide = sh.wide;  // block-uniform
      if (wide) dh_leaf_pairs<false>(sh, sj, diagonal, ni, nj, rule, thr, mine);
      else dh_leaf_pairs<true>(sh, sj, diagonal, ni, nj, rule, thr, mine);
      __syncthreads();
      dh_two_bins(sh, sj, rule, thr, mine);
      if (wide) dh_general<false>(sh, sj, diagonal, ni, nj, rule, mine);
      else dh_general<true>(sh, sj, diagonal, ni, nj, rule, mine);
      __syncthreads();
      dh_unsure(sh, sj, rule, thr, mine);
      ++since;
    }
  }
  if (cur >= 0) dh_flush(hist, nb, counts + (size_t)cur * nb);
}

// Boundary k between bins k and k + 1 is 10 log10 d = k + 1/2; as values of a = sin^2(d / 2R), a margin
// below and above it, rounded outwards. Boundaries past half the circumference are never reached.
void dh_thresholds(int bins, double R, float2* thr) {
  const double pi = 3.14159265358979323846;
  for (int k = 0; k < bins; ++k) {
    float v[2];
    for (int q = 0; q < 2; ++q) {
      const double d = std::pow(10.0, (k + 0.5 + (q ? 1.0 : -1.0) * (double)DH_MARGIN_A) / 10.0);
      const double x = d / (2.0 * R);
      const double s = std::sin(x);
      v[q] = x >= 0.5 * pi ? INFINITY : std::nextafter((float)(s * s), q ? INFINITY : 0.0f);
    }
    thr[k] = make_float2(v[0], v[1]);
  }
}

int dh_fail(lm_ctx* c, int code, const char* msg) {
  if (c) ctx_set_error(c, msg);
  return code;
}

int dh_cuda(lm_ctx* c, cudaError_t e) {
  if (e == cudaSuccess) return LM_OK;
  cudaGetLastError();
  return dh_fail(c, e == cudaErrorMemoryAllocation ? LM_ERR_OOM : LM_ERR_CUDA, cudaGetErrorString(e));
}

}  // namespace
}  // namespace lm

namespace lm {
namespace {

// Carves the call's arrays out of the context's scratch buffer.
struct DhArena {
  unsigned char* base = nullptr;
  size_t used = 0;
  template <class T>
  T* take(size_t n) {
    T* p = reinterpret_cast<T*>(base + used);
    used += (n * sizeof(T) + 255) / 256 * 256;
    return p;
  }
};

// Histograms of n points, either per species (species given, n_seg = 3) or per segment (off).
int dh_run(lm_ctx* c, const float* lat, const float* lon, const int8_t* species, uint32_t n,
           const std::vector<int64_t>& off, uint32_t n_seg, int bins, double radius_m, uint64_t* counts) {
  const size_t nb = (size_t)bins + 1;
  std::vector<DhSeg> hs(n_seg);
  DhCtl hc{};
  hc.box[0] = hc.box[1] = 0xffffffffu;
  uint64_t pstart = 0, n_tiles = 0;
  if (!species) {
    for (uint32_t s = 0; s < n_seg; ++s) {
      const uint32_t m = (uint32_t)(off[s + 1] - off[s]);
      hs[s] = DhSeg{hc.n_items, (uint32_t)off[s], (uint32_t)pstart, m, (uint32_t)n_tiles};
      n_tiles += dh_tiles(m);
      hc.n_items += dh_items(m);
      pstart += dh_padded(m);
    }
    if (pstart > 0xffffffffull) return dh_fail(c, LM_ERR_ARG, "too many segments");
  } else {
    pstart = (uint64_t)n + 3 * DH_LEAF;
    n_tiles = (uint64_t)dh_tiles(n) + 2;  // at most: the counts are known on the device
  }
  int r;
  if ((r = dh_cuda(c, cudaSetDevice(ctx_device(c))))) return r;
  cudaStream_t st = ctx_stream(c);
  // key: segment in the high bits (one more value for points in no segment), place on the curve below
  int seg_bits = 0;
  while (seg_bits < 31 && (n_seg >> seg_bits) != 0) ++seg_bits;
  const int mb = std::min(DH_CURVE_BITS, 32 - seg_bits) & ~1;
  const size_t hl = radix_sort_hist_len(n);
  const size_t out_n = nb * n_seg;
  const ScratchCall scratch(c);
  DhArena ar;
  float *dlat = nullptr, *dlon = nullptr;
  int8_t* dsp = nullptr;
  uint32_t *key = nullptr, *k1 = nullptr, *k2 = nullptr, *v1 = nullptr, *v2 = nullptr, *hist = nullptr,
           *hscan = nullptr, *bsum = nullptr;
  float4 *pts = nullptr, *vec = nullptr;
  DhTile* tiles = nullptr;
  DhSeg* dseg = nullptr;
  DhCtl* dctl = nullptr;
  float2* dthr = nullptr;
  unsigned long long* dcnt = nullptr;
  for (int pass = 0; pass < 2; ++pass) {  // sizes first, then addresses
    ar.used = 0;
    dlat = ar.take<float>(n);
    dlon = ar.take<float>(n);
    dsp = ar.take<int8_t>(species ? n : 0);
    key = ar.take<uint32_t>(n);
    k1 = ar.take<uint32_t>(n);
    k2 = ar.take<uint32_t>(n);
    v1 = ar.take<uint32_t>(n);
    v2 = ar.take<uint32_t>(n);
    hist = ar.take<uint32_t>(hl);
    hscan = ar.take<uint32_t>(hl);
    bsum = ar.take<uint32_t>(SCAN_BLOCKS);
    pts = ar.take<float4>((size_t)pstart);
    vec = ar.take<float4>((size_t)pstart);
    tiles = ar.take<DhTile>((size_t)n_tiles);
    dseg = ar.take<DhSeg>(n_seg);
    dctl = ar.take<DhCtl>(1);
    dthr = ar.take<float2>(bins);
    dcnt = ar.take<unsigned long long>(out_n);
    if (pass == 0) {
      void* p = nullptr;
      if ((r = ctx_scratch(c, ar.used, &p))) return r;
      ar.base = static_cast<unsigned char*>(p);
    }
  }
  DhRule rule{};
  std::vector<float2> thr(bins);
  dh_thresholds(bins, (double)(float)radius_m, thr.data());
  rule.thr = dthr;
  rule.R = (float)radius_m;
  rule.log_2R10 = (float)(10.0 * std::log10(2.0 * (double)rule.R));
  const double smin = std::sin(std::min(1.5 / (2.0 * (double)rule.R), 1.5));
  rule.a_min = (float)(smin * smin);
  rule.bins = bins;
  const char* ex = std::getenv("LM_HIST_EXACT");
  rule.exact = (ex && ex[0] == '1') ? 1 : 0;
  if ((r = dh_cuda(c, cudaMemcpyAsync(dlat, lat, n * sizeof(float), cudaMemcpyHostToDevice, st))) ||
      (r = dh_cuda(c, cudaMemcpyAsync(dlon, lon, n * sizeof(float), cudaMemcpyHostToDevice, st))) ||
      (species && (r = dh_cuda(c, cudaMemcpyAsync(dsp, species, n, cudaMemcpyHostToDevice, st)))) ||
      (!species && (r = dh_cuda(c, cudaMemcpyAsync(dseg, hs.data(), n_seg * sizeof(DhSeg), cudaMemcpyHostToDevice, st)))) ||
      (r = dh_cuda(c, cudaMemcpyAsync(dctl, &hc, sizeof(hc), cudaMemcpyHostToDevice, st))) ||
      (r = dh_cuda(c, cudaMemcpyAsync(dthr, thr.data(), bins * sizeof(float2), cudaMemcpyHostToDevice, st))) ||
      (r = dh_cuda(c, cudaMemsetAsync(dcnt, 0, out_n * sizeof(unsigned long long), st))))
    return r;
  const unsigned blocks_n = (n + 255u) / 256u;
  const unsigned sms = (unsigned)std::max(ctx_sms(c), 1);
  const int8_t* sp = species ? dsp : nullptr;
  k_dh_box<<<std::min(blocks_n, sms * 4u), 256, 0, st>>>(dlat, dlon, sp, n, dctl);
  if (species) k_dh_species_segs<<<1, 1, 0, st>>>(dctl, dseg);
  k_dh_key<<<blocks_n, 256, 0, st>>>(dlat, dlon, sp, n, dseg, n_seg, mb, dctl, key);
  const uint32_t *skey, *sval;
  radix_sort(SortBufs{key, k1, k2, v1, v2, hist, hscan, bsum}, n, std::max(1, mb + seg_bits), st, &skey, &sval);
  k_dh_gather<<<(unsigned)n_tiles, DH_TILE, 0, st>>>(dlat, dlon, sval, dseg, n_seg, pts, vec, tiles);
  const size_t smem = (size_t)DH_WARPS * nb * DH_COPIES * sizeof(uint32_t) + (size_t)bins * sizeof(float2);
  int per_sm = 0;
  if ((r = dh_cuda(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_dist_hist<false>, DH_THREADS, smem))))
    return r;
  // bounds of the items when the counts are on the device (even thirds, one species). With at most half as many as
  // blocks, whole items leave SMs idle: 3,000 points on the globe 368 us so and 207 shared out (357 pair by pair), at
  // one place 470 and 200 (406), 300 on the globe 258 and 162; from 17,000 on, all blocks have items.
  const unsigned long long least = species ? 3 * dh_items(n / 3) : hc.n_items, most = species ? dh_items(n) + 3 : hc.n_items;
  const unsigned long long fit = (unsigned long long)std::max(per_sm, 1) * sms;
  if (2 * least <= fit)
    k_dist_hist<true><<<(unsigned)std::min(most * DH_GROUPS, fit), DH_THREADS, smem, st>>>(pts, vec, tiles, dseg, n_seg,
                                                                                         dctl, rule, dcnt);
  else
    k_dist_hist<false><<<(unsigned)std::min(most, fit), DH_THREADS, smem, st>>>(pts, vec, tiles, dseg, n_seg, dctl, rule,
                                                                                dcnt);
  if ((r = dh_cuda(c, cudaGetLastError()))) return r;
  std::vector<uint64_t> out(out_n);
  if ((r = dh_cuda(c, cudaMemcpyAsync(out.data(), dcnt, out_n * sizeof(uint64_t), cudaMemcpyDeviceToHost, st))) ||
      (r = dh_cuda(c, cudaMemcpyAsync(&hc, dctl, sizeof(hc), cudaMemcpyDeviceToHost, st))) ||
      (r = dh_cuda(c, cudaStreamSynchronize(st))))
    return r;
  if (hc.bad) return dh_fail(c, LM_ERR_NAN, "non-finite coordinates");
  std::copy(out.begin(), out.end(), counts);
  return LM_OK;
}

int dh_check(lm_ctx* c, const float* lat, const float* lon, int64_t n, int bins, double radius_m,
             const uint64_t* counts) {
  if (!counts || (n > 0 && (!lat || !lon))) return dh_fail(c, LM_ERR_ARG, "NULL argument");
  if (n < 0 || n > 0x7fffff00) return dh_fail(c, LM_ERR_ARG, "point count out of range");
  if (bins < 1 || bins > DH_BINS_MAX) return dh_fail(c, LM_ERR_ARG, "bins must be in [1, 256]");
  if (!(radius_m > 0.0) || !std::isfinite(radius_m)) return dh_fail(c, LM_ERR_ARG, "radius must be finite and > 0");
  return LM_OK;
}

}  // namespace
}  // namespace lm

using namespace lm;

extern "C" int lm_distance_histogram(lm_ctx* c, const float* lat, const float* lon, int64_t n, const int64_t* seg,
                                     int n_seg, int bins, double radius_m, uint64_t* counts) {
  if (!c) return LM_ERR_ARG;
  int r;
  if ((r = dh_check(c, lat, lon, n, bins, radius_m, counts))) return r;
  if (n_seg < 1 || (n_seg > 1 && !seg)) return dh_fail(c, LM_ERR_ARG, "n_seg >= 1 and seg offsets are required");
  try {
    std::vector<int64_t> off(n_seg + 1);
    if (seg) {
      for (int s = 0; s <= n_seg; ++s) off[s] = seg[s];
    } else {
      off[0] = 0;
      off[1] = n;
    }
    if (off[0] != 0 || off[n_seg] != n) return dh_fail(c, LM_ERR_ARG, "segments must start at 0 and end at n");
    for (int s = 0; s < n_seg; ++s)
      if (off[s + 1] < off[s]) return dh_fail(c, LM_ERR_ARG, "segment offsets must not decrease");
    if (n == 0) {
      std::fill(counts, counts + ((size_t)bins + 1) * n_seg, (uint64_t)0);
      return LM_OK;
    }
    return dh_run(c, lat, lon, nullptr, (uint32_t)n, off, (uint32_t)n_seg, bins, radius_m, counts);
  } catch (const std::bad_alloc&) {
    return dh_fail(c, LM_ERR_OOM, "out of host memory");
  }
}

extern "C" int lm_species_histogram(lm_ctx* c, const float* lat, const float* lon, const int8_t* species, int64_t n,
                                    int bins, double radius_m, uint64_t* counts) {
  if (!c) return LM_ERR_ARG;
  int r;
  if ((r = dh_check(c, lat, lon, n, bins, radius_m, counts))) return r;
  if (n > 0 && !species) return dh_fail(c, LM_ERR_ARG, "NULL argument");
  if (n == 0) {
    std::fill(counts, counts + 3 * ((size_t)bins + 1), (uint64_t)0);
    return LM_OK;
  }
  try {
    return dh_run(c, lat, lon, species, (uint32_t)n, {}, 3, bins, radius_m, counts);
  } catch (const std::bad_alloc&) {
    return dh_fail(c, LM_ERR_OOM, "out of host memory");
  }
}
