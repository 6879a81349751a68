// The loss of the differentiation benchmark: mean squared great-circle distance between positions and targets, in
// float64, with its derivatives in the same pass (the reference has no differentiation).
//
// Written as tensor operations the loss is some 25 launches forward and 35 backward, most of them waiting for the host:
// 1.2 ms beside the 1.2 ms of 48 recorded steps of 100,000 microbes and their backward. Here it is one pass over the
// positions and a sum of the blocks' parts, in an order fixed by n: 0.54 ms there, nearly all of it in the host's calls
// around it. From some 300,000 positions it is bound by float64 arithmetic (four sincos, an asin, a root, two divisions
// and a reciprocal root a position): 0.3 ms of kernel at 1,000,000.
#include "lm_api.h"
#include "lm_internal.h"

namespace lm {

constexpr int LOSS_THREADS = 256;
constexpr int LOSS_BLOCKS = 152 * 8;  // parts of the sum (LM_LOSS_PARTS)
static_assert(LOSS_BLOCKS <= LM_LOSS_PARTS, "the caller's workspace holds the parts");
constexpr double EARTH_RADIUS_M = 6371.228e3;

// Sum over the block, in thread 0.
__device__ __forceinline__ double block_sum_f64(double v) {
  __shared__ double part[LOSS_THREADS / 32];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0;
  if (threadIdx.x == 0)
    for (int w = 0; w < LOSS_THREADS / 32; ++w) t += part[w];
  return t;
}

// h = sin^2((p2 - p1)/2) + cos p1 cos p2 sin^2((l2 - l1)/2), d = 2 R asin(sqrt(min(h, 1))). The derivative follows the
// chain factor by factor, so it is infinite or undefined where a factor is (d = 0, antipodes) and zero where h > 1.
template <bool GRAD, class T>
__global__ void __launch_bounds__(LOSS_THREADS) k_loss(int64_t n, const double* __restrict__ lon,
                                                       const double* __restrict__ lat, const T* __restrict__ tlon,
                                                       const T* __restrict__ tlat, double* __restrict__ g,
                                                       double* __restrict__ targets, double* __restrict__ part) {
  const double r = 3.14159265358979323846 / 180.0;
  double sum = 0;
  for (int64_t k = blockIdx.x * (int64_t)LOSS_THREADS + threadIdx.x; k < n; k += (int64_t)gridDim.x * LOSS_THREADS) {
    const double l2 = (double)tlon[k], a2 = (double)tlat[k];
    const double p1 = __dmul_rn(lat[k], r), p2 = __dmul_rn(a2, r);  // (a fused p2 - p1 would keep bits of p2 alone)
    double su, cu, sw, cw, s1, c1, s2, c2;
    sincos((p2 - p1) / 2, &su, &cu);
    sincos((l2 - lon[k]) * r / 2, &sw, &cw);
    sincos(p1, &s1, &c1);
    sincos(p2, &s2, &c2);
    const double h = su * su + c1 * c2 * (sw * sw);
    const double q = sqrt(h > 1.0 ? 1.0 : h);
    const double d = 2 * EARTH_RADIUS_M * asin(q);
    sum += d * d;
    if (GRAD) {
      const double ga = 2 * d / (double)n * (2 * EARTH_RADIUS_M) * rsqrt(1.0 - q * q);
      const double gh = h > 1.0 ? 0.0 : ga / (2 * q);
      g[k] = -gh * (c1 * c2) * (sw * cw) * r;
      g[n + k] = -gh * (su * cu + s1 * c2 * (sw * sw)) * r;
      targets[k] = l2;
      targets[n + k] = a2;
    }
  }
  sum = block_sum_f64(sum);
  if (threadIdx.x == 0) part[blockIdx.x] = sum;
}

__global__ void __launch_bounds__(LOSS_THREADS) k_loss_sum(const double* __restrict__ part, int parts, int64_t n,
                                                           double* __restrict__ loss) {
  pdl_wait();
  double v = 0;
  for (int k = threadIdx.x; k < parts; k += LOSS_THREADS) v += part[k];
  v = block_sum_f64(v);
  if (threadIdx.x == 0) *loss = v / (double)n;
}

template <class T>
static void launch_loss(int64_t n, const double* lon, const double* lat, const void* tlon, const void* tlat, double* g,
                        double* targets, double* part, double* loss, cudaStream_t st) {
  const int64_t want = (n + LOSS_THREADS - 1) / LOSS_THREADS;
  const int grid = (int)(want < LOSS_BLOCKS ? want : LOSS_BLOCKS);
  const T *a = static_cast<const T*>(tlon), *o = static_cast<const T*>(tlat);
  if (g)
    k_loss<true, T><<<grid, LOSS_THREADS, 0, st>>>(n, lon, lat, a, o, g, targets, part);
  else
    k_loss<false, T><<<grid, LOSS_THREADS, 0, st>>>(n, lon, lat, a, o, nullptr, nullptr, part);
  launch_dep(k_loss_sum, dim3(1), dim3(LOSS_THREADS), st, (const double*)part, grid, n, loss);
}

}  // namespace lm

extern "C" int lm_mean_squared_distance(int device, uintptr_t stream, int64_t n, const double* lon, const double* lat,
                                        const void* tlon, const void* tlat, int targets_f64, double* loss, double* g,
                                        double* targets, double* work) {
  if (n < 1 || !lon || !lat || !tlon || !tlat || !loss || !work || (g && !targets)) return LM_ERR_ARG;
  int before = 0;
  if (cudaGetDevice(&before) != cudaSuccess || cudaSetDevice(device) != cudaSuccess) return LM_ERR_CUDA;
  const cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (targets_f64)
    lm::launch_loss<double>(n, lon, lat, tlon, tlat, g, targets, work, loss, st);
  else
    lm::launch_loss<float>(n, lon, lat, tlon, tlat, g, targets, work, loss, st);
  const cudaError_t e = cudaGetLastError();
  cudaSetDevice(before);
  return e == cudaSuccess ? LM_OK : LM_ERR_CUDA;
}
