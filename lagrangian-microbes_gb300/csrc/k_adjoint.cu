// K6 + K7: adjoint of the RK4 advection. The reference has no differentiation; the forward scheme
// is the one of K1 (particle_advecter.py:177-187, 220-223), shared through lm_field.cuh so that
// float32 trajectories are bit-identical to lm_step's; in every precision the backward recomputes its own
// forward's.
//
// K6 k_adj_step: one thread per microbe takes x_m (recomputed from a checkpoint) and the adjoint
// lambda_{m+1} = dL/dx_{m+1}, and returns lambda_m by running the four RK4 stages forward and
// their Jacobians backward:
//   x' = x + dt/6 (k1 + 2 k2 + 2 k3 + k4),  k_s = f(t_s, x_s),  f = (U / (M cos lat), V / M),
//   with U, V bilinear in (lon, lat), linear in time, M = 1852 * 60 m per degree.
// For every stage it emits a record (a, b, dL/dU_s, dL/dV_s) for the field cell it sampled: the
// stage's bilinear fractions inside its cell and its adjoint in field units.
//
// K7, the deterministic reduction of the records onto the grid. A cell has 24 sums (two components, three
// stage times, four corners). The terms of a sum are split at fixed powers of two, 2^(22 k), and the
// parts are added as integers, so a sum does not depend on the order of the records and no sort is
// needed; three parts are kept from the largest term down, at least 43 bits below it (FixSum):
//   k_adj_alloc    reserves room for the entries of every occupied cell (K6 counted them) and lists
//                  the cells, in whatever order its blocks come;
//   k_adj_scatter  puts an entry (microbe, which of its stages) into each cell a microbe sampled;
//   k_adj_gather   a warp for every 128 entries of a cell: their sums, put together by the cell's last warp;
//   k_adj_nodes    adds, for every grid node, the four cells around it in a fixed order and spreads the
//                  three stage times onto the field's frames with the linear-in-time weights.
// The gradient is bit-identical from run to run and for every checkpoint interval. A sort of the
// microbes by cell (two radix passes of four launches) with compensated float sums in a fixed order
// took 13 launches a step; here several steps share one set of launches when their records fit L2
// together (a microbe's steps only depend on its own adjoint), and a batch is reduced on a stream of its
// own beside the next one's steps. Forward and backward with the benchmark's loss: 5,000 microbes x 24
// steps in f64 5.96 -> 2.21 ms, 100k x 48 in f32 6.62 -> 1.62 ms, 1M x 24 in ds 7.02 -> 4.10 ms (0.6, 0.7 and
// 0.5 ms of it through the loss in one kernel, k_loss.cu).
#include <algorithm>

#include "lm_field.cuh"
#include "lm_internal.h"

namespace lm {

// Threads per block of the stepping kernels (at most). With 128, the backward step keeps seven blocks an
// SM at 72 registers (a few spills): 1M microbes in double-float, forward and backward of 24 steps, take
// 4.49 ms against 4.75 at its 95 registers (five blocks) and 4.93 with two blocks of 256.
constexpr unsigned ADJ_THREADS = 128;

// ---------------------------------------------------------------- stage table, recompute

// Stage brackets of step m at t_m = t_start + m * dt (the arithmetic of k_step_begin).
__global__ void k_adj_stages(FieldView f, double t_start, double dt, int n_steps, AdjStep* table, uint32_t* err) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= n_steps) return;
  const double t0 = t_start + (double)m * dt;
  const double ts[3] = {t0, t0 + 0.5 * dt, t0 + dt};
  AdjStep s;
  int ok = 1;
  for (int k = 0; k < 3; ++k) {
    const Stage sg = stage_at(f, ts[k]);
    s.k[k] = sg.k;
    s.w[k] = sg.w;
    // the float64 weight of the same bracket (stage_at rounds it to float32)
    const double fk = (ts[k] - f.t0) / f.dT;
    s.wd[k] = sg.w == 0.f ? 0.0 : fmin(fmax(fk - (double)sg.k, 0.0), 1.0);
    ok = ok && sg.ok;
  }
  table[m] = s;
  if (!ok) atomicOr(err, (uint32_t)ERRB_TIME);
}

// Geometry of the offset frame in the working precision T. The float32 instance is the forward
// engine's (FieldView's float fields); the float64 one is the same grid in float64.
template <class T>
struct Geo;
template <>
struct Geo<float> {
  float gx0, gy0, inv_dx, inv_dy, max_fx, max_fy, org_lat;
  __device__ explicit Geo(const FieldView& f)
      : gx0(f.gx0), gy0(f.gy0), inv_dx(f.inv_dx), inv_dy(f.inv_dy), max_fx(f.max_fx), max_fy(f.max_fy),
        org_lat(f.org_lat) {}
};
template <>
struct Geo<double> {
  double gx0, gy0, inv_dx, inv_dy, max_fx, max_fy, org_lat;
  __device__ explicit Geo(const FieldView& f)
      : gx0(f.gx0d), gy0(f.gy0d), inv_dx(f.inv_dxd), inv_dy(f.inv_dyd), max_fx(f.max_fx), max_fy(f.max_fy),
        org_lat((double)f.org_lat) {}
};
__device__ __forceinline__ float cospi_t(float x) { return cospif(x); }
__device__ __forceinline__ double cospi_t(double x) { return cospi(x); }
__device__ __forceinline__ float sinpi_t(float x) { return sinpif(x); }
__device__ __forceinline__ double sinpi_t(double x) { return sinpi(x); }
template <class T>
__device__ __forceinline__ T stage_w(const AdjStep& s, int g);
template <>
__device__ __forceinline__ float stage_w<float>(const AdjStep& s, int g) { return s.w[g]; }
template <>
__device__ __forceinline__ double stage_w<double>(const AdjStep& s, int g) { return s.wd[g]; }

// Absolute float32 positions -> offsets from the field's float32 origin (exact in float64), status.
template <class T>
__global__ void k_adj_init(FieldView f, uint32_t n, const float* __restrict__ lon, const float* __restrict__ lat,
                           T* __restrict__ x, T* __restrict__ y, uint8_t* __restrict__ st) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const float a = lon[p], b = lat[p];
  x[p] = (T)((double)a - (double)f.org_lon);
  y[p] = (T)((double)b - (double)f.org_lat);
  st[p] = (isfinite(a) && isfinite(b)) ? STATUS_OK : STATUS_NAN;
}

template <class T>
__global__ void k_adj_final(FieldView f, uint32_t n, const T* __restrict__ x, const T* __restrict__ y,
                            float* __restrict__ lon, float* __restrict__ lat) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  if (sizeof(T) == sizeof(float)) {  // the engine's rounding of the recorded position
    lon[p] = __fadd_rn(f.org_lon, (float)x[p]);
    lat[p] = __fadd_rn(f.org_lat, (float)y[p]);
  } else {
    lon[p] = (float)((double)f.org_lon + (double)x[p]);
    lat[p] = (float)((double)f.org_lat + (double)y[p]);
  }
}

// Final positions in float64 (absolute degrees) from the T-typed state.
template <class T>
__global__ void k_adj_final64(FieldView f, uint32_t n, const T* __restrict__ x, const T* __restrict__ y,
                              double* __restrict__ lon, double* __restrict__ lat) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  lon[p] = (double)f.org_lon + (double)x[p];
  lat[p] = (double)f.org_lat + (double)y[p];
}

// dL/dx of the final positions (float32) into the T-typed adjoint state, and back out at the end.
template <class T>
__global__ void k_adj_convert_in(uint32_t n, const float* __restrict__ gx, const float* __restrict__ gy,
                                 T* __restrict__ lx, T* __restrict__ ly) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  lx[p] = (T)gx[p];
  ly[p] = (T)gy[p];
}
template <class T>
__global__ void k_adj_convert_out(uint32_t n, const T* __restrict__ lx, const T* __restrict__ ly,
                                  float* __restrict__ gx, float* __restrict__ gy) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  gx[p] = (float)lx[p];
  gy[p] = (float)ly[p];
}

// ---------------------------------------------------------------- K6: one backward step

// Velocity and its Jacobian w.r.t. the offset position. For T = float the value is computed with
// exactly the arithmetic of velocity() so that the recomputed stage positions are the forward's.
template <class T>
struct VelJac {
  T flon, flat;                          // deg/s
  T dlon_dx, dlon_dy, dlat_dx, dlat_dy;  // 1/s
  uint32_t cell;                         // j * (nx - 1) + i
  T a, b;                                // bilinear fractions
  T inv_mc;                              // d flon / d U = 1 / (M cos lat)
};

// Velocity and Jacobian in cell (i, j) at bilinear fractions (a, b); `lat` is the absolute latitude. JAC false: the
// velocity alone (the compiler drops what feeds only the Jacobian, but not the sine that comes with the cosine in
// float64: 3.70 ms a forward of 48 steps of 100,000 microbes with it, 3.46 without).
// sincospi's cosine is cospi's to the last bit (CUDA 13.0, 1.7e7 latitudes compared), so both find the same stages.
template <bool JAC = true, class T>
__device__ __forceinline__ void vel_jac_at(const FieldView& f, int k, T w, int i, int j, T a, T b, T lat, T inv_dx,
                                           T inv_dy, VelJac<T>& r) {
  const float2* p = f.uv + ((size_t)k * f.ny + j) * f.nx + i;
  float2 q00 = __ldg(p), q01 = __ldg(p + 1), q10 = __ldg(p + f.nx), q11 = __ldg(p + f.nx + 1);
  const T w00 = (T(1) - a) * (T(1) - b), w01 = a * (T(1) - b), w10 = (T(1) - a) * b, w11 = a * b;
  T u = w00 * (T)q00.x + w01 * (T)q01.x + w10 * (T)q10.x + w11 * (T)q11.x;
  T v = w00 * (T)q00.y + w01 * (T)q01.y + w10 * (T)q10.y + w11 * (T)q11.y;
  T ua = (T(1) - b) * ((T)q01.x - (T)q00.x) + b * ((T)q11.x - (T)q10.x);
  T ub = (T(1) - a) * ((T)q10.x - (T)q00.x) + a * ((T)q11.x - (T)q01.x);
  T va = (T(1) - b) * ((T)q01.y - (T)q00.y) + b * ((T)q11.y - (T)q10.y);
  T vb = (T(1) - a) * ((T)q10.y - (T)q00.y) + a * ((T)q11.y - (T)q01.y);
  if (w != T(0)) {
    p += (size_t)f.nx * f.ny;
    q00 = __ldg(p); q01 = __ldg(p + 1); q10 = __ldg(p + f.nx); q11 = __ldg(p + f.nx + 1);
    const T u1 = w00 * (T)q00.x + w01 * (T)q01.x + w10 * (T)q10.x + w11 * (T)q11.x;
    const T v1 = w00 * (T)q00.y + w01 * (T)q01.y + w10 * (T)q10.y + w11 * (T)q11.y;
    u = u + w * (u1 - u);
    v = v + w * (v1 - v);
    ua = ua + w * (((T(1) - b) * ((T)q01.x - (T)q00.x) + b * ((T)q11.x - (T)q10.x)) - ua);
    ub = ub + w * (((T(1) - a) * ((T)q10.x - (T)q00.x) + a * ((T)q11.x - (T)q01.x)) - ub);
    va = va + w * (((T(1) - b) * ((T)q01.y - (T)q00.y) + b * ((T)q11.y - (T)q10.y)) - va);
    vb = vb + w * (((T(1) - a) * ((T)q10.y - (T)q00.y) + a * ((T)q11.y - (T)q01.y)) - vb);
  }
  const T M = (T)M_PER_DEG;
  T c, tan_lat;
  if constexpr (sizeof(T) == 8) {  // one argument reduction, one division
    T sn = 0;
    if constexpr (JAC)
      sincospi(lat * (T(1) / T(180)), &sn, &c);
    else
      c = cospi_t(lat * (T(1) / T(180)));
    r.inv_mc = T(1) / (M * c);
    r.flon = u * r.inv_mc;
    tan_lat = sn * M * r.inv_mc;
  } else {  // the forward's operations
    c = cospi_t(lat * (T(1) / T(180)));
    r.flon = u / (M * c);
    r.inv_mc = T(1) / (M * c);
    tan_lat = sinpi_t(lat * (T(1) / T(180))) / c;
  }
  r.flat = v * (T(1) / M);
  // d/dlat (1 / cos(lat)) = tan(lat) / cos(lat) * pi / 180 per degree
  r.dlon_dx = ua * inv_dx * r.inv_mc;
  r.dlon_dy = ub * inv_dy * r.inv_mc + r.flon * tan_lat * (T)0.017453292519943295;
  r.dlat_dx = va * inv_dx * (T(1) / M);
  r.dlat_dy = vb * inv_dy * (T(1) / M);
  r.cell = (uint32_t)j * (uint32_t)(f.nx - 1) + (uint32_t)i;
  r.a = a;
  r.b = b;
}

template <bool JAC = true, class T>
__device__ __forceinline__ bool vel_jac(const FieldView& f, const Geo<T>& g, int k, T w, T xo, T yo, VelJac<T>& r) {
  const T fx = (xo - g.gx0) * g.inv_dx;
  const T fy = (yo - g.gy0) * g.inv_dy;
  if (!(fx >= T(0) && fx <= g.max_fx && fy >= T(0) && fy <= g.max_fy)) return false;
  const int i = min((int)fx, f.nx - 2);
  const int j = min((int)fy, f.ny - 2);
  vel_jac_at<JAC>(f, k, w, i, j, fx - (T)i, fy - (T)j, g.org_lat + yo, g.inv_dx, g.inv_dy, r);
  return true;
}

// One RK4 step in precision T. For T = float it is rk4_step, the engine's own arithmetic.
template <class T>
__device__ __forceinline__ bool rk4_t(const FieldView& f, const Geo<T>& g, const AdjStep& s, T dt, T x, T y, T& nx,
                                      T& ny);
template <>
__device__ __forceinline__ bool rk4_t<float>(const FieldView& f, const Geo<float>&, const AdjStep& s, float dt, float x,
                                             float y, float& nx, float& ny) {
  const Stage sh[3] = {{s.k[0], s.w[0], 1}, {s.k[1], s.w[1], 1}, {s.k[2], s.w[2], 1}};
  return rk4_step(f, f.uv, sh, dt, x, y, nx, ny);
}
template <>
__device__ __forceinline__ bool rk4_t<double>(const FieldView& f, const Geo<double>& g, const AdjStep& s, double dt,
                                              double x, double y, double& nx, double& ny) {
  VelJac<double> J1, J2, J3, J4;
  bool ok = vel_jac<false>(f, g, s.k[0], s.wd[0], x, y, J1);
  ok = ok && vel_jac<false>(f, g, s.k[1], s.wd[1], x + 0.5 * dt * J1.flon, y + 0.5 * dt * J1.flat, J2);
  ok = ok && vel_jac<false>(f, g, s.k[1], s.wd[1], x + 0.5 * dt * J2.flon, y + 0.5 * dt * J2.flat, J3);
  ok = ok && vel_jac<false>(f, g, s.k[2], s.wd[2], x + dt * J3.flon, y + dt * J3.flat, J4);
  if (!ok) return false;
  nx = x + (J1.flon + 2.0 * J2.flon + 2.0 * J3.flon + J4.flon) * (dt * (1.0 / 6.0));
  ny = y + (J1.flat + 2.0 * J2.flat + 2.0 * J3.flat + J4.flat) * (dt * (1.0 / 6.0));
  return true;
}

// Steps [m0, m1) of every microbe in registers, the forward's freezing rules. With rec_* set, the
// state before every step is stored ([m - m0][n]) for the backward sweep.
template <class T>
__global__ void __launch_bounds__(ADJ_THREADS) k_adj_forward(FieldView f, const AdjStep* __restrict__ table, int m0, int m1,
                                                     T dt, uint32_t n, T* __restrict__ xs, T* __restrict__ ys,
                                                     uint8_t* __restrict__ sts, T* __restrict__ rec_x,
                                                     T* __restrict__ rec_y, uint8_t* __restrict__ rec_st,
                                                     uint32_t* err) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const Geo<T> g(f);
  T x = xs[p], y = ys[p];
  uint8_t st = sts[p];
  uint32_t bits = 0;
  for (int m = m0; m < m1; ++m) {
    if (rec_x) {
      const size_t o = (size_t)(m - m0) * n + p;
      rec_x[o] = x;
      rec_y[o] = y;
      rec_st[o] = st;
    }
    if (st != STATUS_OK) continue;
    const AdjStep s = table[m];
    T nx, ny;
    if (rk4_t<T>(f, g, s, dt, x, y, nx, ny)) {
      if (isfinite(nx) && isfinite(ny)) {
        x = nx;
        y = ny;
      } else {
        st = STATUS_NAN;
        bits |= ERRB_NAN;
      }
    } else {
      st = (isfinite(x) && isfinite(y)) ? STATUS_OOB : STATUS_NAN;
      bits |= st == STATUS_OOB ? (uint32_t)ERRB_OOB : (uint32_t)ERRB_NAN;
    }
  }
  xs[p] = x;
  ys[p] = y;
  sts[p] = st;
  if (bits) atomicOr(err, bits);
}

// The backward of one RK4 step of microbe p from its four stage Jacobians (every precision):
// lambda_{m+1} -> lambda_m in gx, gy, plus its 4 records.
template <class T>
__device__ __forceinline__ void adj_tail(const VelJac<T>* J, T dt, T& gx, T& gy, float4* __restrict__ rec) {
  const T h6 = dt * (T(1) / T(6)), h3 = dt * (T(1) / T(3)), h2 = T(0.5) * dt;
  // dL/dk4, then back through x3 = x + dt k3, x2 = x + dt/2 k2, x1 = x + dt/2 k1
  const T g4x = h6 * gx, g4y = h6 * gy;
  const T x3x = J[3].dlon_dx * g4x + J[3].dlat_dx * g4y, x3y = J[3].dlon_dy * g4x + J[3].dlat_dy * g4y;
  const T g3x = h3 * gx + dt * x3x, g3y = h3 * gy + dt * x3y;
  const T x2x = J[2].dlon_dx * g3x + J[2].dlat_dx * g3y, x2y = J[2].dlon_dy * g3x + J[2].dlat_dy * g3y;
  const T g2x = h3 * gx + h2 * x2x, g2y = h3 * gy + h2 * x2y;
  const T x1x = J[1].dlon_dx * g2x + J[1].dlat_dx * g2y, x1y = J[1].dlon_dy * g2x + J[1].dlat_dy * g2y;
  const T g1x = h6 * gx + h2 * x1x, g1y = h6 * gy + h2 * x1y;
  const T x0x = J[0].dlon_dx * g1x + J[0].dlat_dx * g1y, x0y = J[0].dlon_dy * g1x + J[0].dlat_dy * g1y;
  gx = gx + ((x0x + x1x) + (x2x + x3x));
  gy = gy + ((x0y + x1y) + (x2y + x3y));
  // records: dL/dU_s = dL/dk_s,lon / (M cos lat_s), dL/dV_s = dL/dk_s,lat / M (float32 for the reduction)
  const T invM = T(1) / (T)M_PER_DEG;
  rec[0] = make_float4((float)J[0].a, (float)J[0].b, (float)(g1x * J[0].inv_mc), (float)(g1y * invM));
  rec[1] = make_float4((float)J[1].a, (float)J[1].b, (float)(g2x * J[1].inv_mc), (float)(g2y * invM));
  rec[2] = make_float4((float)J[2].a, (float)J[2].b, (float)(g3x * J[2].inv_mc), (float)(g3y * invM));
  rec[3] = make_float4((float)J[3].a, (float)J[3].b, (float)(g4x * J[3].inv_mc), (float)(g4y * invM));
}

// A microbe has one entry in every cell its stages sampled: the stages of that cell as bits. The cell
// of stage 1 comes first; which of the stages 2..4 open another entry, and its bits.
__device__ __forceinline__ uint32_t base_mask(const uint4& c) {
  return 1u | (c.y == c.x ? 2u : 0u) | (c.z == c.x ? 4u : 0u) | (c.w == c.x ? 8u : 0u);
}
template <class F>
__device__ __forceinline__ void for_other_cells(const uint4& c, F&& f) {
  if (c.y != c.x) f(c.y, 2u | (c.z == c.y ? 4u : 0u) | (c.w == c.y ? 8u : 0u));
  if (c.z != c.x && c.z != c.y) f(c.z, 4u | (c.w == c.z ? 8u : 0u));
  if (c.w != c.x && c.w != c.y && c.w != c.z) f(c.w, 8u);
}

// Count the entries of one microbe's step (every lane of the warp calls this; `ok` false: no entries). Lanes
// with the same first cell, the usual case, share the atomic.
__device__ __forceinline__ void count_entries(const AdjBatch& b, int q, bool ok, const uint4& c) {
  uint32_t* count = b.count + (size_t)q * b.cells;
  const uint32_t peers = __match_any_sync(0xffffffffu, ok ? c.x : NONE);
  if (!ok) return;
  if ((threadIdx.x & 31u) == (uint32_t)(__ffs(peers) - 1)) atomicAdd(count + c.x, (uint32_t)__popc(peers));
  for_other_cells(c, [&](uint32_t cell, uint32_t) { atomicAdd(count + cell, 1u); });
}

// Steps m_last, m_last - 1, ... (`steps` of them) of every microbe: lambda_{m+1} -> lambda_m, plus 4
// records and the 4 stage cells a step. A frozen step (a stage left the grid or the step was
// non-finite, as in the forward) passes the adjoint through and has no entries. xs, ys, sts: the
// states before step m at offset (m - m_last) * n.
template <class T>
__global__ void __launch_bounds__(ADJ_THREADS, sizeof(T) == 8 ? 1 : 7) k_adj_step(FieldView f, const AdjStep* __restrict__ table, int m_last, T dt,
                                                  AdjBatch b, const T* __restrict__ xs, const T* __restrict__ ys,
                                                  const uint8_t* __restrict__ sts, T* __restrict__ lx,
                                                  T* __restrict__ ly) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = p < b.n;
  const Geo<T> g(f);
  T gx = live ? lx[p] : T(0), gy = live ? ly[p] : T(0);
  for (int q = 0; q < b.steps; ++q) {
    const AdjStep s = table[m_last - q];
    const ptrdiff_t o = (ptrdiff_t)p - (ptrdiff_t)q * b.n;
    const T w0 = stage_w<T>(s, 0), w1 = stage_w<T>(s, 1), w2 = stage_w<T>(s, 2);
    VelJac<T> J[4];
    bool ok = live && sts[o] == STATUS_OK;
    uint4 c = make_uint4(NONE, NONE, NONE, NONE);
    if (ok) {
      const T x = xs[o], y = ys[o];
      ok = ok && vel_jac(f, g, s.k[0], w0, x, y, J[0]);
      ok = ok && vel_jac(f, g, s.k[1], w1, x + T(0.5) * dt * J[0].flon, y + T(0.5) * dt * J[0].flat, J[1]);
      ok = ok && vel_jac(f, g, s.k[1], w1, x + T(0.5) * dt * J[1].flon, y + T(0.5) * dt * J[1].flat, J[2]);
      ok = ok && vel_jac(f, g, s.k[2], w2, x + dt * J[2].flon, y + dt * J[2].flat, J[3]);
      if (ok) {
        const T nx = x + (J[0].flon + T(2) * J[1].flon + T(2) * J[2].flon + J[3].flon) * (dt * (T(1) / T(6)));
        const T ny = y + (J[0].flat + T(2) * J[1].flat + T(2) * J[2].flat + J[3].flat) * (dt * (T(1) / T(6)));
        ok = isfinite(nx) && isfinite(ny);
      }
      if (ok) {
        adj_tail<T>(J, dt, gx, gy, b.rec + 4 * ((size_t)q * b.n + p));
        c = make_uint4(J[0].cell, J[1].cell, J[2].cell, J[3].cell);
      }
    }
    if (live) b.cell[(size_t)q * b.n + p] = c;
    count_entries(b, q, ok, c);
  }
  if (live) {
    lx[p] = gx;
    ly[p] = gy;
  }
}

// ---------------------------------------------------------------- double-float positions
//
// The default working precision of the tape (ADJ_DS): each offset is an unevaluated sum of two
// float32 words, hi + lo (about 48 significant bits), so a 720-step trajectory does not pick up the
// float32 rounding of the position every step (0.1 m at the field's scale) that the flow then
// amplifies. Only the position arithmetic is double-float: stage positions, the RK4 update and the
// position -> (cell, bilinear fraction) mapping. Velocities, Jacobians, the adjoint state and the
// records stay float32 with the f32 mode's arithmetic (vel_jac_at<float>). Error-free sums and
// products follow Dekker (1971) and Knuth's two-sum; every operation is rounded explicitly
// (__fadd_rn & co.) so that no contraction changes it between kernels.
struct DS {
  float hi, lo;
};

__device__ __forceinline__ DS ds_of(double d) {
  const float h = (float)d;
  return DS{h, (float)(d - (double)h)};
}
__device__ __forceinline__ double ds_value(DS a) { return (double)a.hi + (double)a.lo; }
__device__ __forceinline__ bool ds_finite(DS a) { return isfinite(a.hi) && isfinite(a.lo); }

// hi + lo of s + t where |s| >= |t| (fast two-sum)
__device__ __forceinline__ DS ds_renorm(float s, float t) {
  const float h = __fadd_rn(s, t);
  return DS{h, __fsub_rn(t, __fsub_rn(h, s))};
}
// a + b, b a float32 (two-sum of the high words, then the low word)
__device__ __forceinline__ DS ds_add(DS a, float b) {
  const float s = __fadd_rn(a.hi, b);
  const float bb = __fsub_rn(s, a.hi);
  const float e = __fadd_rn(__fsub_rn(a.hi, __fsub_rn(s, bb)), __fsub_rn(b, bb));
  return ds_renorm(s, __fadd_rn(e, a.lo));
}
// a + b for two double-float values
__device__ __forceinline__ DS ds_add(DS a, DS b) {
  const float s = __fadd_rn(a.hi, b.hi);
  const float bb = __fsub_rn(s, a.hi);
  const float e = __fadd_rn(__fsub_rn(a.hi, __fsub_rn(s, bb)), __fsub_rn(b.hi, bb));
  return ds_renorm(s, __fadd_rn(e, __fadd_rn(a.lo, b.lo)));
}
// a * b (the product of the high words is exact through one fma)
__device__ __forceinline__ DS ds_mul(DS a, DS b) {
  const float p = __fmul_rn(a.hi, b.hi);
  float e = __fmaf_rn(a.hi, b.hi, -p);
  e = __fmaf_rn(a.hi, b.lo, e);
  e = __fmaf_rn(a.lo, b.hi, e);
  return ds_renorm(p, e);
}

// The grid in double-float: fx = (x - gx0) / dx with 1/dx to double-float accuracy (a float32
// 1/dx alone would shift the sampling point by up to ~0.1 m at the far edge of the grid).
struct GeoDS {
  // (split into two words on the host: twelve float64 operations a thread took a quarter of the time of
  // a backward step)
  DS mgx0, mgy0, inv_dx, inv_dy;  // -gx0, -gy0 (grid origin minus state origin), 1/dx, 1/dy
  float max_fx, max_fy, org_lat, inv_dxf, inv_dyf;
  __device__ explicit GeoDS(const FieldView& f)
      : mgx0{f.ds_mgx0.x, f.ds_mgx0.y}, mgy0{f.ds_mgy0.x, f.ds_mgy0.y}, inv_dx{f.ds_inv_dx.x, f.ds_inv_dx.y},
        inv_dy{f.ds_inv_dy.x, f.ds_inv_dy.y}, max_fx(f.max_fx), max_fy(f.max_fy), org_lat(f.org_lat),
        inv_dxf(f.inv_dx), inv_dyf(f.inv_dy) {}
};

// Cell index and bilinear fraction of a double-float grid coordinate u in [0, max]; false outside.
__device__ __forceinline__ bool ds_cell(DS u, float max_u, int n_cells, int& i, float& a) {
  const bool in = (u.hi > 0.f || (u.hi == 0.f && u.lo >= 0.f)) && (u.hi < max_u || (u.hi == max_u && u.lo <= 0.f));
  if (!in) return false;
  float fl = floorf(u.hi);
  if (fl == u.hi && u.lo < 0.f) fl = __fsub_rn(fl, 1.f);  // hi is an integer and the value lies just below it
  i = min((int)fl, n_cells - 1);
  a = __fadd_rn(__fsub_rn(u.hi, (float)i), u.lo);  // u.hi - i is exact (Sterbenz) for i >= 1, and for i = 0
  return true;
}

// Velocity and Jacobian at a double-float offset position (float32 arithmetic past the fractions).
__device__ __forceinline__ bool vel_jac_ds(const FieldView& f, const GeoDS& g, int k, float w, DS xo, DS yo,
                                           VelJac<float>& r) {
  int i, j;
  float a, b;
  if (!ds_cell(ds_mul(ds_add(xo, g.mgx0), g.inv_dx), g.max_fx, f.nx - 1, i, a)) return false;
  if (!ds_cell(ds_mul(ds_add(yo, g.mgy0), g.inv_dy), g.max_fy, f.ny - 1, j, b)) return false;
  vel_jac_at(f, k, w, i, j, a, b, __fadd_rn(g.org_lat, yo.hi), g.inv_dxf, g.inv_dyf, r);
  return true;
}

// The increment (k1 + 2 k2 + 2 k3 + k4) dt / 6 of one coordinate, float32.
__device__ __forceinline__ float rk4_increment(float k1, float k2, float k3, float k4, float dt) {
  return __fmul_rn(__fadd_rn(__fadd_rn(k1, __fmul_rn(2.f, k2)), __fadd_rn(__fmul_rn(2.f, k3), k4)), dt * (1.0f / 6.0f));
}

// Stage q (0..3) of one RK4 step from (x, y): its velocity and Jacobian in J[q], given the earlier
// stages J[0..q-1] (stage positions x + dt/2 k1, x + dt/2 k2, x + dt k3). False outside the grid.
// The forward, the backward recomputation and the cell signature all evaluate stages through this.
__device__ __forceinline__ bool ds_stage(const FieldView& f, const GeoDS& g, const AdjStep& s, float dt, DS x, DS y,
                                         VelJac<float>* J, int q) {
  if (q == 0) return vel_jac_ds(f, g, s.k[0], s.w[0], x, y, J[0]);
  const float h = q == 3 ? dt : 0.5f * dt;
  const int g_ = q == 3 ? 2 : 1;
  return vel_jac_ds(f, g, s.k[g_], s.w[g_], ds_add(x, __fmul_rn(h, J[q - 1].flon)), ds_add(y, __fmul_rn(h, J[q - 1].flat)),
                    J[q]);
}

// One RK4 step from (x, y): the four stages and the new position. False when a stage leaves the grid.
__device__ __forceinline__ bool rk4_ds(const FieldView& f, const GeoDS& g, const AdjStep& s, float dt, DS x, DS y,
                                       VelJac<float>* J, DS& nx, DS& ny) {
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (!ds_stage(f, g, s, dt, x, y, J, q)) return false;
  nx = ds_add(x, rk4_increment(J[0].flon, J[1].flon, J[2].flon, J[3].flon, dt));
  ny = ds_add(y, rk4_increment(J[0].flat, J[1].flat, J[2].flat, J[3].flat, dt));
  return true;
}

__global__ void k_adj_init_ds(FieldView f, uint32_t n, const float* __restrict__ lon, const float* __restrict__ lat,
                              DS* __restrict__ x, DS* __restrict__ y, uint8_t* __restrict__ st) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const float a = lon[p], b = lat[p];
  x[p] = ds_of((double)a - (double)f.org_lon);
  y[p] = ds_of((double)b - (double)f.org_lat);
  st[p] = (isfinite(a) && isfinite(b)) ? STATUS_OK : STATUS_NAN;
}

__global__ void k_adj_final_ds(FieldView f, uint32_t n, const DS* __restrict__ x, const DS* __restrict__ y,
                               float* __restrict__ lon, float* __restrict__ lat, double* __restrict__ lon64,
                               double* __restrict__ lat64) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const double a = (double)f.org_lon + ds_value(x[p]), b = (double)f.org_lat + ds_value(y[p]);
  if (lon) {
    lon[p] = (float)a;
    lat[p] = (float)b;
  } else {
    lon64[p] = a;
    lat64[p] = b;
  }
}

__global__ void __launch_bounds__(ADJ_THREADS) k_adj_forward_ds(FieldView f, const AdjStep* __restrict__ table, int m0, int m1,
                                                        float dt, uint32_t n, DS* __restrict__ xs, DS* __restrict__ ys,
                                                        uint8_t* __restrict__ sts, DS* __restrict__ rec_x,
                                                        DS* __restrict__ rec_y, uint8_t* __restrict__ rec_st,
                                                        uint32_t* err) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const GeoDS g(f);
  DS x = xs[p], y = ys[p];
  uint8_t st = sts[p];
  uint32_t bits = 0;
  for (int m = m0; m < m1; ++m) {
    if (rec_x) {
      const size_t o = (size_t)(m - m0) * n + p;
      rec_x[o] = x;
      rec_y[o] = y;
      rec_st[o] = st;
    }
    if (st != STATUS_OK) continue;
    VelJac<float> J[4];
    DS nx, ny;
    if (rk4_ds(f, g, table[m], dt, x, y, J, nx, ny)) {
      if (ds_finite(nx) && ds_finite(ny)) {
        x = nx;
        y = ny;
      } else {
        st = STATUS_NAN;
        bits |= ERRB_NAN;
      }
    } else {
      st = (ds_finite(x) && ds_finite(y)) ? STATUS_OOB : STATUS_NAN;
      bits |= st == STATUS_OOB ? (uint32_t)ERRB_OOB : (uint32_t)ERRB_NAN;
    }
  }
  xs[p] = x;
  ys[p] = y;
  sts[p] = st;
  if (bits) atomicOr(err, bits);
}

__global__ void __launch_bounds__(ADJ_THREADS, 7) k_adj_step_ds(FieldView f, const AdjStep* __restrict__ table, int m_last,
                                                     float dt, AdjBatch b, const DS* __restrict__ xs,
                                                     const DS* __restrict__ ys, const uint8_t* __restrict__ sts,
                                                     float* __restrict__ lx, float* __restrict__ ly) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = p < b.n;
  const GeoDS g(f);
  float gx = live ? lx[p] : 0.f, gy = live ? ly[p] : 0.f;
  for (int q = 0; q < b.steps; ++q) {
    const AdjStep s = table[m_last - q];
    const ptrdiff_t o = (ptrdiff_t)p - (ptrdiff_t)q * b.n;
    VelJac<float> J[4];
    bool ok = live && sts[o] == STATUS_OK;
    uint4 c = make_uint4(NONE, NONE, NONE, NONE);
    if (ok) {
      DS nx, ny;
      ok = rk4_ds(f, g, s, dt, xs[o], ys[o], J, nx, ny) && ds_finite(nx) && ds_finite(ny);
      if (ok) {
        adj_tail<float>(J, dt, gx, gy, b.rec + 4 * ((size_t)q * b.n + p));
        c = make_uint4(J[0].cell, J[1].cell, J[2].cell, J[3].cell);
      }
    }
    if (live) b.cell[(size_t)q * b.n + p] = c;
    count_entries(b, q, ok, c);
  }
  if (live) {
    lx[p] = gx;
    ly[p] = gy;
  }
}

__global__ void __launch_bounds__(256) k_adj_signature_ds(FieldView f, const AdjStep* __restrict__ table, int n_steps,
                                                          float dt, uint32_t n, const DS* __restrict__ xs,
                                                          const DS* __restrict__ ys, const uint8_t* __restrict__ sts,
                                                          unsigned long long* __restrict__ sig) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const GeoDS g(f);
  DS x = xs[p], y = ys[p];
  bool live = sts[p] == STATUS_OK;
  unsigned long long h = 0;
  const unsigned long long nx = (unsigned long long)f.nx, cw = (unsigned long long)(f.nx - 1);
  for (int m = 0; m < n_steps && live; ++m) {
    const AdjStep s = table[m];
    VelJac<float> J[4];
    int q = 0;
#pragma unroll
    for (; q < 4; ++q) {  // the stages evaluated, up to one that leaves the grid
      if (!ds_stage(f, g, s, dt, x, y, J, q)) break;
      h = (h ^ ((J[q].cell / cw) * nx + J[q].cell % cw)) * 0x100000001B3ull;
    }
    if (q < 4) break;
    const DS x1 = ds_add(x, rk4_increment(J[0].flon, J[1].flon, J[2].flon, J[3].flon, dt));
    const DS y1 = ds_add(y, rk4_increment(J[0].flat, J[1].flat, J[2].flat, J[3].flat, dt));
    if (!(ds_finite(x1) && ds_finite(y1))) break;
    x = x1;
    y = y1;
  }
  sig[p] = h;
}

// Cell path of every microbe over steps [0, n_steps): the grid cell (j * nx + i) of each stage that
// the forward evaluated, folded in order as sig = (sig ^ cell) * 0x100000001B3. The stage
// positions come from vel_jac, whose values are the forward's; two runs of one microbe with equal
// signatures sampled the same bilinear pieces, so the map between them is smooth.
template <class T>
__global__ void __launch_bounds__(256) k_adj_signature(FieldView f, const AdjStep* __restrict__ table, int n_steps,
                                                       T dt, uint32_t n, const T* __restrict__ xs,
                                                       const T* __restrict__ ys, const uint8_t* __restrict__ sts,
                                                       unsigned long long* __restrict__ sig) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const Geo<T> g(f);
  T x = xs[p], y = ys[p];
  bool live = sts[p] == STATUS_OK;
  unsigned long long h = 0;
  const unsigned long long nx = (unsigned long long)f.nx, cw = (unsigned long long)(f.nx - 1);
  for (int m = 0; m < n_steps && live; ++m) {
    const AdjStep s = table[m];
    const int ks[4] = {s.k[0], s.k[1], s.k[1], s.k[2]};
    const T ws[4] = {stage_w<T>(s, 0), stage_w<T>(s, 1), stage_w<T>(s, 1), stage_w<T>(s, 2)};
    const T hs[4] = {T(0), T(0.5), T(0.5), T(1)};
    T kx[4], ky[4];
    bool ok = true;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (!ok) break;
      VelJac<T> J;
      const T sx = q == 0 ? x : x + hs[q] * dt * kx[q - 1];
      const T sy = q == 0 ? y : y + hs[q] * dt * ky[q - 1];
      ok = vel_jac<false>(f, g, ks[q], ws[q], sx, sy, J);
      if (ok) {
        h = (h ^ ((J.cell / cw) * nx + J.cell % cw)) * 0x100000001B3ull;
        kx[q] = J.flon;
        ky[q] = J.flat;
      }
    }
    if (!ok) break;
    const T nx_ = x + (kx[0] + T(2) * kx[1] + T(2) * kx[2] + kx[3]) * (dt * (T(1) / T(6)));
    const T ny_ = y + (ky[0] + T(2) * ky[1] + T(2) * ky[2] + ky[3]) * (dt * (T(1) / T(6)));
    if (!(isfinite(nx_) && isfinite(ny_))) break;
    x = nx_;
    y = ny_;
  }
  sig[p] = h;
}

// ---------------------------------------------------------------- K7: reduction onto the grid

// Entries of an item of a cell of m entries (a multiple of ADJ_ITEM).
__device__ __forceinline__ uint32_t item_size(uint32_t m) {
  return ADJ_ITEM * max(1u, m / (ADJ_ITEM * ADJ_SPLIT) + (m % (ADJ_ITEM * ADJ_SPLIT) ? 1u : 0u));
}

// Room for the entries of every occupied cell of step blockIdx.y (consecutive from place[c]), the list of
// items and room for the parts of cells of several items: one reservation of each per block.
constexpr int ALLOC_THREADS = 512;
__global__ void __launch_bounds__(ALLOC_THREADS) k_adj_alloc(AdjBatch b) {
  pdl_wait();
  __shared__ uint32_t ws[3][ALLOC_THREADS / 32], base[3];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t c = blockIdx.x * ALLOC_THREADS + threadIdx.x;
  const size_t o = (size_t)blockIdx.y * b.cells;
  const uint32_t m = c < b.cells ? b.count[o + c] : 0u, size = item_size(m), items = m / size + (m % size ? 1u : 0u);
  const uint32_t parts = items > 1 ? items : 0u;
  uint32_t sum[3] = {m, items, parts};  // inclusive sums over the warp
  for (int d = 1; d < 32; d <<= 1) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const uint32_t x = __shfl_up_sync(0xffffffffu, sum[k], d);
      if (lane >= (uint32_t)d) sum[k] += x;
    }
  }
  if (lane == 31)
    for (int k = 0; k < 3; ++k) ws[k][warp] = sum[k];
  __syncthreads();
  if (threadIdx.x < 3) {
    uint32_t* w = ws[threadIdx.x];
    uint32_t t = 0;
    for (int k = 0; k < ALLOC_THREADS / 32; ++k) {
      const uint32_t x = w[k];
      w[k] = t;
      t += x;
    }
    base[threadIdx.x] = t ? atomicAdd(b.total + 4 * blockIdx.y + threadIdx.x, t) : 0u;
  }
  __syncthreads();
  if (!m) return;
  const uint32_t at = base[0] + ws[0][warp] + sum[0] - m;
  const uint32_t part = base[2] + ws[2][warp] + sum[2] - parts;
  b.place[o + c] = at;
  uint4* list = b.list + (size_t)blockIdx.y * adj_items(b.n, b.cells) + base[1] + ws[1][warp] + sum[1] - items;
  for (uint32_t k = 0; k < items; ++k)
    list[k] = make_uint4(c, at + k * size, min(size, m - k * size), parts ? part + k : NONE);
  uint32_t* done = b.done + (size_t)blockIdx.y * adj_parts(b.n) + part;
  for (uint32_t k = 0; k < parts; ++k) done[k] = 0u;
}

// Entries of the microbes' steps into their cells, in whatever order they come.
__global__ void __launch_bounds__(256) k_adj_scatter(AdjBatch b) {
  pdl_wait();
  const uint32_t p = blockIdx.x * 256 + threadIdx.x, lane = threadIdx.x & 31u;
  const uint32_t q = blockIdx.y;
  uint32_t* place = b.place + (size_t)q * b.cells;
  uint2* ent = b.ent + (size_t)q * 4 * b.n;
  const uint4 c = p < b.n ? b.cell[(size_t)q * b.n + p] : make_uint4(NONE, NONE, NONE, NONE);
  const uint32_t peers = __match_any_sync(0xffffffffu, c.x);
  if (c.x == NONE) return;
  const int leader = __ffs(peers) - 1;
  uint32_t at = 0;
  if (lane == (uint32_t)leader) at = atomicAdd(place + c.x, (uint32_t)__popc(peers));
  at = __shfl_sync(peers, at, leader) + __popc(peers & ((1u << lane) - 1u));
  ent[at] = make_uint2(p, base_mask(c));
  for_other_cells(c, [&](uint32_t cell, uint32_t mask) { ent[atomicAdd(place + cell, 1u)] = make_uint2(p, mask); });
}

// Sum of float32 terms as three integers. A term is split at the fixed powers of two 2^(22 k): its part in
// units of 2^(22 k) is the rest of the parts above, rounded to the nearest integer, so in any unit above it
// a term is 0 and its parts do not depend on where the splitting starts. The sum keeps three units, from
// the first in which the largest term has at most 21 bits (`top`) down: 43 bits below that term at least,
// where the term itself was rounded 24 below. (One scale for the 24 sums of a cell, two parts below the
// largest adjoint of all, lost the small terms of a corner beside a large adjoint elsewhere in the cell:
// 1e-2 of the sum at a ratio of 1e-10.) Adding 1.5 * 2^23 leaves the integer in a float's low bits, and
// the sums run on the raw bits (the constant is taken out at the end).
constexpr float FIX_MAGIC = 12582912.0f, FIX_UNIT = 4194304.0f;  // 1.5 * 2^23, 2^22
struct FixSum {
  uint32_t a, b, c;
};
__device__ __forceinline__ void fix_add(FixSum& s, float v, float scale) {
  const float t = fmaf(v, scale, FIX_MAGIC);
  const float r = fmaf(v, scale, FIX_MAGIC - t);  // exact, in [-1/2, 1/2]
  const float t1 = fmaf(r, FIX_UNIT, FIX_MAGIC);
  const float r1 = fmaf(r, FIX_UNIT, FIX_MAGIC - t1);  // exact
  s.a += __float_as_uint(t);
  s.b += __float_as_uint(t1);
  s.c += __float_as_uint(fmaf(r1, FIX_UNIT, FIX_MAGIC));
}
// The first unit of terms up to the one of float bits `most` is 2^(22 (top - 6)): 1 <= top <= 11 (from 1, the
// last unit lies below the smallest float). Its reciprocal.
__device__ __forceinline__ uint32_t fix_top(uint32_t most) { return max(((most >> 23) + 6u) / 22u, 1u); }
__device__ __forceinline__ float fix_scale(uint32_t top) { return __uint_as_float((259u - 22u * top) << 23); }

// A sum that is infinite or undefined: `top` is FIX_SPECIAL, and a says which of the terms were there.
constexpr uint32_t FIX_SPECIAL = 15u, FIX_NAN = 1u, FIX_PLUS = 2u, FIX_MINUS = 4u;
__device__ __forceinline__ uint32_t fix_flags(float v) {
  return isfinite(v) ? 0u : isnan(v) ? FIX_NAN : v > 0.f ? FIX_PLUS : FIX_MINUS;
}

// (a 2^44 + b 2^22 + c) units of the last place of `top`, rounded once.
__device__ __forceinline__ float fix_value(uint32_t top, long long a, long long b, long long c) {
  if (top == FIX_SPECIAL)
    return ((uint32_t)a & FIX_NAN) || (a & (FIX_PLUS | FIX_MINUS)) == (FIX_PLUS | FIX_MINUS) ? NAN
           : a & FIX_PLUS                                                                   ? INFINITY
                                                                                            : -INFINITY;
  b += c >> 22;
  a += b >> 22;
  const long long low = (b & 0x3fffffll) << 22 | (c & 0x3fffffll);  // in [0, 2^44)
  const long long mag = a < 0 ? -a : a;
  int e = 22 * ((int)top - 6) - 44;
  long long x;  // at least 41 bits, or all of them; what is cut off leaves its mark in the last bit
  if (mag < 1ll << 18) {
    x = (a << 44) + low;
  } else if (mag < 1ll << 32) {
    x = ((a << 29) + (low >> 15)) | (low & 0x7fffll ? 1ll : 0ll);
    e += 15;
  } else {
    x = ((a << 8) + (low >> 36)) | (low & 0xfffffffffll ? 1ll : 0ll);
    e += 36;
  }
  return ldexpf(__ll2float_rn(x), e);
}

// Eight values of every lane combined over the lanes of the same last two bits: lane l gets value
// (l >> 4 & 1) * 4 + (l >> 3 & 1) * 2 + (l >> 2 & 1). Every step halves what a lane keeps. Lanes of last
// bits 1 and 2 (the two stages at t + dt/2) then get each other's too.
template <class F>
__device__ __forceinline__ uint32_t by_stage(const uint32_t (&in)[8], F&& op) {
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t v[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = in[i];
#pragma unroll
  for (int h = 4; h > 0; h >>= 1) {
    const bool upper = (lane & (4u * h)) != 0u;
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const uint32_t send = upper ? v[i] : v[i + h], keep = upper ? v[i + h] : v[i];
      v[i] = op(keep, __shfl_xor_sync(0xffffffffu, send, 4 * h));
    }
  }
  const uint32_t other = __shfl_xor_sync(0xffffffffu, v[0], 3), s = lane & 3u;
  return s == 1u || s == 2u ? op(v[0], other) : v[0];
}

// The terms of a record: corners (00, 01, 10, 11) of dL/dU, then of dL/dV.
template <class F>
__device__ __forceinline__ void for_terms(const float4& r, F&& f) {
  const float a = r.x, b = r.y;
  const float w[4] = {(1.f - a) * (1.f - b), a * (1.f - b), (1.f - a) * b, a * b};
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    f(q, w[q] * r.z);
    f(4 + q, w[q] * r.w);
  }
}

// A sum in parts of its own `top`, and another one added to it: the parts below the larger top's last unit
// are dropped from either (there they are the same integers whatever the sum's other terms).
struct FixTotal {
  uint32_t top = 0u;
  long long a = 0, b = 0, c = 0;
  __device__ __forceinline__ void join(uint32_t t, long long xa, long long xb, long long xc) {
    if (t == FIX_SPECIAL || top == FIX_SPECIAL) {
      a = (top == FIX_SPECIAL ? a : 0ll) | (t == FIX_SPECIAL ? xa : 0ll);
      top = FIX_SPECIAL;
      return;
    }
    const uint32_t up = t > top ? t - top : 0u, down = t < top ? top - t : 0u;
    if (up) {
      c = up == 1u ? b : up == 2u ? a : 0ll;
      b = up == 1u ? a : 0ll;
      a = 0ll;
      top = t;
    }
    a += down == 0u ? xa : 0ll;
    b += down == 0u ? xb : down == 1u ? xa : 0ll;
    c += down == 0u ? xc : down == 1u ? xb : down == 2u ? xa : 0ll;
  }
  __device__ __forceinline__ float value() const { return fix_value(top, a, b, c); }
};

// The sums of an item, or of several: [3][24], a lane's own at `part`.
constexpr uint32_t PART_GROUP = 32;
static_assert(ADJ_SPLIT <= PART_GROUP * PART_GROUP, "two levels put a cell's items together");
__device__ __forceinline__ void part_store(long long* part, uint32_t slot, const FixTotal& t, bool on) {
  long long* p = part + (size_t)slot * 72;
  if (on) {
    p[0] = t.a * 16 + t.top;  // (|a| < 2^54)
    p[24] = t.b;
    p[48] = t.c;
  }
  __threadfence();
  __syncwarp();
}
// Is this the last of n warps to come here? (whole warp; the others' parts can be read then)
__device__ __forceinline__ bool part_last(uint32_t* done, uint32_t n) {
  uint32_t before = 0;
  if ((threadIdx.x & 31u) == 0) before = atomicAdd(done, 1u);
  const bool last = __shfl_sync(0xffffffffu, before, 0) == n - 1u;
  if (last) __threadfence();
  return last;
}
__device__ __noinline__ FixTotal part_merge(const long long* p, uint32_t stride, uint32_t n) {
  FixTotal total;
  for (uint32_t k0 = 0; k0 < n; k0 += 4) {
    long long x[4][3];
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
#pragma unroll
      for (uint32_t j = 0; j < 3; ++j) x[k][j] = k0 + k < n ? __ldcg(p + (size_t)(k0 + k) * stride + 24 * j) : 0ll;
    }
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) total.join((uint32_t)x[k][0] & 15u, x[k][0] >> 4, x[k][1], x[k][2]);
  }
  return total;
}

// A warp per item: four lanes take an entry, one each of its stages (stage 1 at t, 2 and 3 at t + dt/2, 4 at
// t + dt), so a warp reads the records of eight entries at a time and holds those of ADJ_CHUNK in
// registers: the largest terms first, then the sums. The items of a cell of several leave their sums in
// `part`, and the warps that finish last put them together (in integers, whichever they are).
// Bound by instruction issue (64 % of the slots; the rest is latency of the records' loads): 47 us a step for
// 1M microbes, where two parts a term, scaled by the cell's largest adjoint, took 35 and kept too few bits
// (the counting of the largest by k_adj_step took 18 us more there: 66 -> 48). Forward and backward of 24
// such steps: chunks of 32 entries at four blocks an SM 4.13 ms, at three 4.20, at five (spills) 4.28, chunks
// of 64 at three 4.21; items of 64 4.22, of 256 4.38; the records read twice (69 us) 4.69. In crowded cells
// the putting together counts: 8 steps of 1M microbes in 56 cells 2.98 ms, in one 23.2, by one warp for all
// items of 128; 2.22 and 2.71 in two levels with at most 1,024 items (256 items: 2.22 and 3.92).
constexpr int GATHER_THREADS = 256, GATHER_BLOCKS = 4;  // threads a block, blocks an SM
constexpr uint32_t ADJ_ROUNDS = 4, ADJ_CHUNK = 8 * ADJ_ROUNDS;
__global__ void __launch_bounds__(GATHER_THREADS, GATHER_BLOCKS) k_adj_gather(AdjBatch b) {
  pdl_wait();
  const uint32_t lane = threadIdx.x & 31u, s = lane & 3u, q = blockIdx.y;
  const uint32_t nt = b.total[4 * q + 1];
  const size_t oc = (size_t)q * b.cells;
  const uint4* list = b.list + (size_t)q * adj_items(b.n, b.cells);
  const uint2* ent = b.ent + (size_t)q * 4 * b.n;
  const float4* rec = b.rec + (size_t)q * 4 * b.n;
  // where this lane's sum goes: stage time, then by_stage's value (lanes of last bits 2 hold the same as those of 1)
  const uint32_t at = (s == 0u ? 0u : s == 3u ? 16u : 8u) + ((lane >> 4 & 1u) * 4u + (lane >> 3 & 1u) * 2u + (lane >> 2 & 1u));
  long long* part = b.part + (size_t)q * adj_parts(b.n) * 72 + at;
  const uint32_t stride = gridDim.x * (GATHER_THREADS / 32);
  uint32_t t = blockIdx.x * (GATHER_THREADS / 32) + (threadIdx.x >> 5);
  uint4 next = t < nt ? list[t] : make_uint4(0u, 0u, 0u, 0u);
  for (; t < nt; t += stride) {
    const uint4 item = next;
    next = t + stride < nt ? list[t + stride] : item;
    const uint32_t c = item.x, lo = item.y, m = item.z;
    FixTotal total;
    for (uint32_t k0 = 0; k0 < m; k0 += ADJ_CHUNK) {
      uint2 e[ADJ_ROUNDS];
      float4 r[ADJ_ROUNDS];
#pragma unroll
      for (uint32_t k = 0; k < ADJ_ROUNDS; ++k) {
        const uint32_t i = k0 + 8u * k + (lane >> 2);
        e[k] = i < m ? ent[lo + i] : make_uint2(0u, 0u);
      }
      uint32_t bits = 0u;  // of the largest adjoint (NaN above infinity above every number)
#pragma unroll
      for (uint32_t k = 0; k < ADJ_ROUNDS; ++k) {
        r[k] = (e[k].y >> s) & 1u ? rec[4 * (size_t)e[k].x + s] : make_float4(0.f, 0.f, 0.f, 0.f);
        bits = max(bits, max(__float_as_uint(r[k].z) & 0x7fffffffu, __float_as_uint(r[k].w) & 0x7fffffffu));
      }
      const uint32_t rounds = (m - k0 + 7u) / 8u;  // with entries; the records of the others add zeros
      uint32_t v[8];
      float most[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) most[k] = 0.f;
#pragma unroll
      for (uint32_t k = 0; k < ADJ_ROUNDS; k += 2) {
        if (k >= rounds) break;
        for_terms(r[k], [&](int i, float x) { most[i] = fmaxf(most[i], fabsf(x)); });
        for_terms(r[k + 1], [&](int i, float x) { most[i] = fmaxf(most[i], fabsf(x)); });
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = __float_as_uint(most[k]);
      const uint32_t top = fix_top(by_stage(v, [](uint32_t x, uint32_t y) { return max(x, y); }));
      uint32_t flags = 0u;
      if (__any_sync(0xffffffffu, bits >= 0x7f800000u)) {
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = 0u;
#pragma unroll
        for (uint32_t k = 0; k < ADJ_ROUNDS; ++k) for_terms(r[k], [&](int i, float x) { v[i] |= fix_flags(x); });
        flags = by_stage(v, [](uint32_t x, uint32_t y) { return x | y; });
      }
      const float own = fix_scale(top);
      float scale[8];
#pragma unroll
      for (int k = 0; k < 8; ++k)
        scale[k] = __shfl_sync(0xffffffffu, own, (k & 4) << 2 | (k & 2) << 2 | (k & 1) << 2 | (int)s);
      FixSum sum[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) sum[k].a = sum[k].b = sum[k].c = 0u;
#pragma unroll
      for (uint32_t k = 0; k < ADJ_ROUNDS; k += 2) {
        if (k >= rounds) break;
        for_terms(r[k], [&](int i, float x) { fix_add(sum[i], x, scale[i]); });
        for_terms(r[k + 1], [&](int i, float x) { fix_add(sum[i], x, scale[i]); });
      }
      const uint32_t magic = min((rounds + 1u) & ~1u, ADJ_ROUNDS) * __float_as_uint(FIX_MAGIC);
      auto add = [](uint32_t x, uint32_t y) { return x + y; };
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = sum[k].a - magic;
      const uint32_t sa = by_stage(v, add);  // at most 2 * ADJ_CHUNK terms of 2^21
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = sum[k].b - magic;
      const uint32_t sb = by_stage(v, add);
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = sum[k].c - magic;
      const uint32_t sc = by_stage(v, add);
      total.join(flags ? FIX_SPECIAL : top, (int)(flags ? flags : sa), (int)sb, (int)sc);
    }
    float* out = b.csum + (oc + c) * 24 + at;
    if (item.w == NONE) {
      if (s != 2u) *out = total.value();
      continue;
    }
    const uint32_t all = b.count[oc + c], size = item_size(all), items = all / size + (all % size ? 1u : 0u);
    const uint32_t index = (lo - (b.place[oc + c] - all)) / size;  // of this item (place: past the cell's last entry)
    // up to PART_GROUP items are put together by the last of them, and up to as many groups by the last group
    const uint32_t first = item.w - index, head = first + index / PART_GROUP * PART_GROUP;
    uint32_t* done = b.done + (size_t)q * adj_parts(b.n);
    part_store(part, item.w, total, s != 2u);
    if (!part_last(done + head, min(PART_GROUP, first + items - head))) continue;
    total = part_merge(part + (size_t)head * 72, 72, min(PART_GROUP, first + items - head));
    if (items > PART_GROUP) {
      part_store(part, head, total, s != 2u);
      const uint32_t groups = (items + PART_GROUP - 1) / PART_GROUP;
      if (!part_last(done + first + 1, groups)) continue;  // (a place that no group counts in)
      total = part_merge(part + (size_t)first * 72, 72 * PART_GROUP, groups);
    }
    if (s != 2u) *out = total.value();
  }
}

// The sums of a batch onto the grid: a block takes 32 consecutive nodes, its warp w step w of every
// blockDim.y steps. The four cells around a node in a fixed order give its sums at the three stage
// times; the first warp then spreads them onto frames k_g (weight 1 - w_g) and k_g + 1 (weight w_g) and
// adds them to the gradient, the steps in turn.
constexpr int NODE_STEPS = 8;
__global__ void __launch_bounds__(32 * NODE_STEPS) k_adj_nodes(int nx, int ny, const AdjStep* __restrict__ table,
                                                               int m_last, AdjBatch b, float* __restrict__ gu,
                                                               float* __restrict__ gv) {
  pdl_wait();
  __shared__ float sums[NODE_STEPS][6][32];
  __shared__ uint32_t busy[NODE_STEPS];  // nodes with sums at the step
  const uint32_t lane = threadIdx.x, w = threadIdx.y;
  const uint32_t node = blockIdx.x * 32 + lane;
  const bool in = node < (uint32_t)nx * (uint32_t)ny;
  const int ni = (int)(node % (uint32_t)nx), nj = (int)(node / (uint32_t)nx);
  const int cw = nx - 1;
  // cell (ci, cj) sees this node as corner (nj - cj) * 2 + (ni - ci)
  const int ci_[4] = {ni - 1, ni, ni - 1, ni}, cj_[4] = {nj - 1, nj - 1, nj, nj}, corner[4] = {3, 2, 1, 0};
  for (int q0 = 0; q0 < b.steps; q0 += (int)blockDim.y) {
    const int q = q0 + (int)w;
    float U[3] = {0.f, 0.f, 0.f}, V[3] = {0.f, 0.f, 0.f};
    if (in && q < b.steps) {
      uint32_t m[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int ci = ci_[t], cj = cj_[t];
        const bool cell = !(ci < 0 || cj < 0 || ci > nx - 2 || cj > ny - 2);
        m[t] = cell ? b.count[(size_t)q * b.cells + (size_t)cj * cw + ci] : 0u;
      }
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        if (m[t] == 0u) continue;  // only cells with entries were summed
        const float* cs = b.csum + ((size_t)q * b.cells + (size_t)cj_[t] * cw + ci_[t]) * 24 + corner[t];
#pragma unroll
        for (int g = 0; g < 3; ++g) {
          U[g] += cs[g * 8];
          V[g] += cs[g * 8 + 4];
        }
      }
    }
    const bool any = !(U[0] == 0.f && U[1] == 0.f && U[2] == 0.f && V[0] == 0.f && V[1] == 0.f && V[2] == 0.f);
    const uint32_t mask = __ballot_sync(0xffffffffu, any);
    if (lane == 0) busy[w] = mask;
    if (any) {
#pragma unroll
      for (int g = 0; g < 3; ++g) {
        sums[w][g][lane] = U[g];
        sums[w][3 + g][lane] = V[g];
      }
    }
    __syncthreads();
    if (w == 0) {
      for (int k = 0; k < (int)blockDim.y; ++k) {
        if (!((busy[k] >> lane) & 1u)) continue;
        const AdjStep s = table[m_last - q0 - k];
        int kmin = s.k[0], kmax = s.k[0];
#pragma unroll
        for (int g = 0; g < 3; ++g) {
          kmin = min(kmin, s.k[g]);
          kmax = max(kmax, s.k[g] + (s.w[g] != 0.f ? 1 : 0));
        }
        const size_t plane = (size_t)nx * ny;
        for (int fr = kmin; fr <= kmax; ++fr) {
          float du = 0.f, dv = 0.f;
          bool hit = false;
#pragma unroll
          for (int g = 0; g < 3; ++g) {
            const float u = sums[k][g][lane], v = sums[k][3 + g][lane];
            if (s.k[g] == fr) {
              du += (1.f - s.w[g]) * u;
              dv += (1.f - s.w[g]) * v;
              hit = true;
            }
            if (s.w[g] != 0.f && s.k[g] + 1 == fr) {
              du += s.w[g] * u;
              dv += s.w[g] * v;
              hit = true;
            }
          }
          if (hit) {
            gu[(size_t)fr * plane + node] += du;
            gv[(size_t)fr * plane + node] += dv;
          }
        }
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------- launchers

static inline unsigned grid_for(size_t n, unsigned block) { return (unsigned)((n + block - 1) / block); }

// ADJ_THREADS, or fewer when that leaves SMs without a block (down to a warp). In float64 it matters
// most: an SM's two float64 lanes are shared by the warps on it (5,000 microbes: 50 -> 24 us a step).
static inline unsigned adj_threads(uint32_t n) {
  unsigned threads = ADJ_THREADS;
  while (threads > 32 && grid_for(n, threads) < 152) threads /= 2;
  return threads;
}

void launch_adj_stages(const FieldView& f, double t_start, double dt, int n_steps, AdjStep* table, uint32_t* err,
                       cudaStream_t st) {
  if (n_steps > 0) k_adj_stages<<<grid_for(n_steps, 128), 128, 0, st>>>(f, t_start, dt, n_steps, table, err);
}

void launch_adj_init(const FieldView& f, int prec, uint32_t n, const float* lon, const float* lat, void* x, void* y,
                     uint8_t* status, cudaStream_t st) {
  if (!n) return;
  if (prec == ADJ_F64)
    k_adj_init<double><<<grid_for(n, 256), 256, 0, st>>>(f, n, lon, lat, (double*)x, (double*)y, status);
  else if (prec == ADJ_DS)
    k_adj_init_ds<<<grid_for(n, 256), 256, 0, st>>>(f, n, lon, lat, (DS*)x, (DS*)y, status);
  else
    k_adj_init<float><<<grid_for(n, 256), 256, 0, st>>>(f, n, lon, lat, (float*)x, (float*)y, status);
}

void launch_adj_final(const FieldView& f, int prec, uint32_t n, const void* x, const void* y, float* lon, float* lat,
                      cudaStream_t st) {
  if (!n) return;
  if (prec == ADJ_F64)
    k_adj_final<double><<<grid_for(n, 256), 256, 0, st>>>(f, n, (const double*)x, (const double*)y, lon, lat);
  else if (prec == ADJ_DS)
    k_adj_final_ds<<<grid_for(n, 256), 256, 0, st>>>(f, n, (const DS*)x, (const DS*)y, lon, lat, nullptr, nullptr);
  else
    k_adj_final<float><<<grid_for(n, 256), 256, 0, st>>>(f, n, (const float*)x, (const float*)y, lon, lat);
}

void launch_adj_final64(const FieldView& f, int prec, uint32_t n, const void* x, const void* y, double* lon,
                        double* lat, cudaStream_t st) {
  if (!n) return;
  if (prec == ADJ_F64)
    k_adj_final64<double><<<grid_for(n, 256), 256, 0, st>>>(f, n, (const double*)x, (const double*)y, lon, lat);
  else if (prec == ADJ_DS)
    k_adj_final_ds<<<grid_for(n, 256), 256, 0, st>>>(f, n, (const DS*)x, (const DS*)y, nullptr, nullptr, lon, lat);
  else
    k_adj_final64<float><<<grid_for(n, 256), 256, 0, st>>>(f, n, (const float*)x, (const float*)y, lon, lat);
}

void launch_adj_seed(int prec, uint32_t n, const float* gx, const float* gy, void* lx, void* ly, cudaStream_t st) {
  if (!n) return;
  if (prec == ADJ_F64)
    k_adj_convert_in<double><<<grid_for(n, 256), 256, 0, st>>>(n, gx, gy, (double*)lx, (double*)ly);
  else
    k_adj_convert_in<float><<<grid_for(n, 256), 256, 0, st>>>(n, gx, gy, (float*)lx, (float*)ly);
}

void launch_adj_unseed(int prec, uint32_t n, const void* lx, const void* ly, float* gx, float* gy, cudaStream_t st) {
  if (!n) return;
  if (prec == ADJ_F64)
    k_adj_convert_out<double><<<grid_for(n, 256), 256, 0, st>>>(n, (const double*)lx, (const double*)ly, gx, gy);
  else
    k_adj_convert_out<float><<<grid_for(n, 256), 256, 0, st>>>(n, (const float*)lx, (const float*)ly, gx, gy);
}

void launch_adj_forward(const FieldView& f, int prec, const AdjStep* table, int m0, int m1, double dt, uint32_t n,
                        void* x, void* y, uint8_t* status, void* rec_x, void* rec_y, uint8_t* rec_st, uint32_t* err,
                        cudaStream_t st) {
  if (!n || m1 <= m0) return;
  const unsigned threads = adj_threads(n), blocks = grid_for(n, threads);
  if (prec == ADJ_F64)
    k_adj_forward<double><<<blocks, threads, 0, st>>>(f, table, m0, m1, dt, n, (double*)x, (double*)y, status,
                                                            (double*)rec_x, (double*)rec_y, rec_st, err);
  else if (prec == ADJ_DS)
    k_adj_forward_ds<<<blocks, threads, 0, st>>>(f, table, m0, m1, (float)dt, n, (DS*)x, (DS*)y, status,
                                                       (DS*)rec_x, (DS*)rec_y, rec_st, err);
  else
    k_adj_forward<float><<<blocks, threads, 0, st>>>(f, table, m0, m1, (float)dt, n, (float*)x, (float*)y, status,
                                                           (float*)rec_x, (float*)rec_y, rec_st, err);
}

void launch_adj_step(const FieldView& f, int prec, const AdjStep* table, int m_last, double dt, const AdjBatch& b,
                     const void* x, const void* y, const uint8_t* status, void* lx, void* ly, cudaStream_t st) {
  if (!b.n) return;
  const unsigned threads = adj_threads(b.n), blocks = grid_for(b.n, threads);
  if (prec == ADJ_F64)
    k_adj_step<double><<<blocks, threads, 0, st>>>(f, table, m_last, dt, b, (const double*)x, (const double*)y, status,
                                                   (double*)lx, (double*)ly);
  else if (prec == ADJ_DS)
    k_adj_step_ds<<<blocks, threads, 0, st>>>(f, table, m_last, (float)dt, b, (const DS*)x, (const DS*)y, status,
                                              (float*)lx, (float*)ly);
  else
    k_adj_step<float><<<blocks, threads, 0, st>>>(f, table, m_last, (float)dt, b, (const float*)x, (const float*)y,
                                                  status, (float*)lx, (float*)ly);
}

void launch_adj_reduce(int nx, int ny, const AdjStep* table, int m_last, const AdjBatch& b, float* gu, float* gv,
                       int sms, cudaStream_t st) {
  if (!b.n) return;
  const unsigned steps = (unsigned)b.steps;
  launch_dep(k_adj_alloc, dim3(grid_for(b.cells, ALLOC_THREADS), steps), dim3(ALLOC_THREADS), st, b);
  launch_dep(k_adj_scatter, dim3(grid_for(b.n, 256), steps), dim3(256), st, b);
  // a warp per item, at most GATHER_BLOCKS blocks an SM over all steps
  const unsigned cap = std::max(1u, (unsigned)(sms > 0 ? sms : 152) * GATHER_BLOCKS / steps);
  const unsigned want = grid_for(adj_items(b.n, b.cells) * 32, GATHER_THREADS);
  launch_dep(k_adj_gather, dim3(std::min(want, cap), steps), dim3(GATHER_THREADS), st, b);
  launch_dep(k_adj_nodes, dim3(grid_for((size_t)nx * ny, 32)), dim3(32, std::min(b.steps, NODE_STEPS)), st, nx, ny, table, m_last, b, gu, gv);
}

void launch_adj_signature(const FieldView& f, int prec, const AdjStep* table, int n_steps, double dt, uint32_t n,
                          const void* x, const void* y, const uint8_t* status, unsigned long long* sig,
                          cudaStream_t st) {
  if (!n) return;
  if (prec == ADJ_F64)
    k_adj_signature<double><<<grid_for(n, 256), 256, 0, st>>>(f, table, n_steps, dt, n, (const double*)x,
                                                              (const double*)y, status, sig);
  else if (prec == ADJ_DS)
    k_adj_signature_ds<<<grid_for(n, 256), 256, 0, st>>>(f, table, n_steps, (float)dt, n, (const DS*)x, (const DS*)y,
                                                         status, sig);
  else
    k_adj_signature<float><<<grid_for(n, 256), 256, 0, st>>>(f, table, n_steps, (float)dt, n, (const float*)x,
                                                             (const float*)y, status, sig);
}

}  // namespace lm
