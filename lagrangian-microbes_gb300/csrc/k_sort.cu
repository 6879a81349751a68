// Stable LSD radix sort of 32-bit keys with their input indices, and the exclusive scan it uses (the
// point order of the distance histogram, the row offsets of pair queries).
#include "lm_internal.h"

namespace lm {

constexpr int RS_THREADS = 256;
constexpr int RS_ITEMS = 16;
constexpr uint32_t RS_TILE = RS_THREADS * RS_ITEMS;
constexpr int RS_WARPS = RS_THREADS / 32;

// Digit histogram of one tile, written digit-major: hist[d * tiles + tile].
__global__ void __launch_bounds__(RS_THREADS) k_rs_hist(const uint32_t* __restrict__ keys, uint32_t m, int shift,
                                                        int bits, uint32_t* __restrict__ hist, uint32_t tiles) {
  __shared__ uint32_t h[RS_RADIX_MAX];
  const uint32_t R = 1u << bits, mask = R - 1u;
  for (uint32_t d = threadIdx.x; d < R; d += RS_THREADS) h[d] = 0;
  __syncthreads();
  const uint32_t base = blockIdx.x * RS_TILE;
  const uint32_t lane = threadIdx.x & 31u;
  for (int r = 0; r < RS_ITEMS; ++r) {
    const uint32_t i = base + (uint32_t)r * RS_THREADS + threadIdx.x;
    const bool valid = i < m;
    const uint32_t d = valid ? (keys[i] >> shift) & mask : R;
    const uint32_t peers = __match_any_sync(0xffffffffu, d);
    if (valid && (peers & ((1u << lane) - 1u)) == 0) atomicAdd(&h[d], (uint32_t)__popc(peers));
  }
  __syncthreads();
  for (uint32_t d = threadIdx.x; d < R; d += RS_THREADS) hist[(size_t)d * tiles + blockIdx.x] = h[d];
}

// Stable scatter of one tile. Warp w takes the tile's w-th run of RS_ITEMS * 32 consecutive items
// (RS_ITEMS rounds of 32) and ranks each item among the equal digits of its run with match masks and
// a per-warp digit counter, without block barriers; the block then turns the counters into per-warp
// digit offsets (the tile's offset of the digit plus the counts of the earlier warps), and each
// item goes to its warp's offset plus its rank: equal keys keep their order.
__global__ void __launch_bounds__(RS_THREADS) k_rs_scatter(const uint32_t* __restrict__ kin,
                                                           const uint32_t* __restrict__ vin,
                                                           uint32_t* __restrict__ kout, uint32_t* __restrict__ vout,
                                                           uint32_t m, int shift, int bits,
                                                           const uint32_t* __restrict__ hscan, uint32_t tiles) {
  __shared__ uint32_t wcnt[RS_WARPS][RS_RADIX_MAX];
  const uint32_t R = 1u << bits, mask = R - 1u;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  for (uint32_t d = threadIdx.x; d < R; d += RS_THREADS)
    for (int w = 0; w < RS_WARPS; ++w) wcnt[w][d] = 0;
  __syncthreads();
  const uint32_t base = blockIdx.x * RS_TILE + warp * (RS_ITEMS * 32u);
  const uint32_t lt = (1u << lane) - 1u;
  uint32_t kk[RS_ITEMS], rk[RS_ITEMS];
#pragma unroll
  for (int r = 0; r < RS_ITEMS; ++r) {
    const uint32_t i = base + (uint32_t)r * 32u + lane;
    const bool valid = i < m;
    const uint32_t k = valid ? kin[i] : 0u;
    const uint32_t d = valid ? (k >> shift) & mask : R;
    const uint32_t peers = __match_any_sync(0xffffffffu, d);
    const uint32_t below = peers & lt;
    const uint32_t c = valid ? wcnt[warp][d] : 0u;  // every peer reads the count before the update
    __syncwarp();
    if (valid && below == 0) wcnt[warp][d] = c + (uint32_t)__popc(peers);
    __syncwarp();
    kk[r] = k;
    rk[r] = c + (uint32_t)__popc(below);
  }
  __syncthreads();
  for (uint32_t d = threadIdx.x; d < R; d += RS_THREADS) {
    uint32_t o = hscan[(size_t)d * tiles + blockIdx.x];
    for (int w = 0; w < RS_WARPS; ++w) {
      const uint32_t c = wcnt[w][d];
      wcnt[w][d] = o;
      o += c;
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < RS_ITEMS; ++r) {
    const uint32_t i = base + (uint32_t)r * 32u + lane;
    if (i < m) {
      const uint32_t o = wcnt[warp][(kk[r] >> shift) & mask] + rk[r];
      kout[o] = kk[r];
      vout[o] = vin ? vin[i] : i;
    }
  }
}

// Exclusive scan of n uint32 values (in -> out), in SCAN_BLOCKS contiguous chunks: block sums, then
// each block adds the sums of the blocks before it while scanning its chunk.
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* sh, uint32_t* total) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t x = v;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= (uint32_t)o) x += y;
  }
  if (lane == 31) sh[warp] = x;
  __syncthreads();
  if (warp == 0) {
    uint32_t s = lane < blockDim.x / 32 ? sh[lane] : 0u;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= (uint32_t)o) s += y;
    }
    sh[lane] = s;  // inclusive warp totals
  }
  __syncthreads();
  const uint32_t before = warp ? sh[warp - 1] : 0u;
  *total = sh[blockDim.x / 32 - 1];
  __syncthreads();
  return before + x - v;
}

__global__ void __launch_bounds__(256) k_scan_sums(const uint32_t* __restrict__ in, size_t n, size_t chunk,
                                                   uint32_t* __restrict__ bsum) {
  __shared__ uint32_t red[8];
  const size_t lo = (size_t)blockIdx.x * chunk, hi = min(n, lo + chunk);
  uint32_t s = 0;
  for (size_t i = lo + threadIdx.x; i < hi; i += blockDim.x) s += in[i];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t t = 0;
    for (int w = 0; w < 8; ++w) t += red[w];
    bsum[blockIdx.x] = t;
  }
}

__global__ void __launch_bounds__(256) k_scan_chunks(const uint32_t* __restrict__ in, uint32_t* __restrict__ out,
                                                     size_t n, size_t chunk, const uint32_t* __restrict__ bsum) {
  __shared__ uint32_t sh[32];
  __shared__ uint32_t carry;
  if (threadIdx.x < 32) {
    uint32_t s = 0;
    for (uint32_t b = threadIdx.x; b < blockIdx.x; b += 32) s += bsum[b];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) carry = s;
  }
  __syncthreads();
  const size_t lo = (size_t)blockIdx.x * chunk, hi = min(n, lo + chunk);
  for (size_t t = lo; t < hi; t += blockDim.x) {
    const size_t i = t + threadIdx.x;
    const uint32_t v = i < hi ? in[i] : 0u;
    uint32_t total;
    const uint32_t ex = block_exclusive_scan(v, sh, &total);
    if (i < hi) out[i] = carry + ex;
    __syncthreads();
    if (threadIdx.x == 0) carry += total;
    __syncthreads();
  }
}

static inline unsigned grid_for(size_t n, unsigned long long block) { return (unsigned)((n + block - 1) / block); }

void launch_scan(const uint32_t* in, uint32_t* out, size_t n, uint32_t* bsum, cudaStream_t st) {
  if (!n) return;
  const size_t chunk = (n + SCAN_BLOCKS - 1) / SCAN_BLOCKS;
  const unsigned nb = grid_for(n, chunk);
  k_scan_sums<<<nb, 256, 0, st>>>(in, n, chunk, bsum);
  k_scan_chunks<<<nb, 256, 0, st>>>(in, out, n, chunk, bsum);
}

size_t radix_sort_hist_len(uint32_t m) { return (size_t)RS_RADIX_MAX * grid_for(m, RS_TILE); }

void radix_sort(const SortBufs& sb, uint32_t m, int key_bits, cudaStream_t st, const uint32_t** skey,
              const uint32_t** sval) {
  const uint32_t tiles = grid_for(m, RS_TILE);
  const int passes = key_bits <= RS_BITS_MAX ? 1 : (key_bits + RS_BITS_MAX - 1) / RS_BITS_MAX;
  const int width = (key_bits + passes - 1) / passes;
  const uint32_t* kin = sb.key;
  const uint32_t* vin = nullptr;
  for (int p = 0; p < passes; ++p) {
    uint32_t* kout = (p & 1) ? sb.k2 : sb.k1;
    uint32_t* vout = (p & 1) ? sb.v2 : sb.v1;
    const int shift = p * width;
    const int bits = key_bits - shift < width ? key_bits - shift : width;
    k_rs_hist<<<tiles, RS_THREADS, 0, st>>>(kin, m, shift, bits, sb.hist, tiles);
    launch_scan(sb.hist, sb.hscan, ((size_t)1 << bits) * tiles, sb.bsum, st);
    k_rs_scatter<<<tiles, RS_THREADS, 0, st>>>(kin, vin, kout, vout, m, shift, bits, sb.hscan, tiles);
    kin = kout;
    vin = vout;
  }
  *skey = kin;
  *sval = vin;
}

}  // namespace lm
