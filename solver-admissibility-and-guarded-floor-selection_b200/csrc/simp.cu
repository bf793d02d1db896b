// SIMP loop kernels around the guarded solve: the cone density filter, its
// transpose, and the optimality-criteria (OC) update.
//
// The reference filters with a row-normalised sparse matrix
// (gpu_fem/pub_simp_solver.py:90-117 _build_density_filter: weight
// rmin - dist for every element within distance < rmin, the element itself
// weight rmin, rows divided by their sums) and runs the OC bisection with one
// SpMV per step (gpu_fem/simp_gpu.py:212-294 _oc_step_cupy).  On the structured
// grid the filter is a stencil over the offsets within rmin, applied here
// directly (row sums from the in-grid offsets), and without a Heaviside
// projection the bisection's volume sum(H rn) equals sum_j (H^T 1)_j rn_j, so a
// bisection step is one fused pass over the design variables.
//
// Element index e = (i * ny + j) * nz + k.  Reductions are deterministic: every
// block writes a partial, one block sums them in block order.
#include <algorithm>
#include <stdexcept>

#include "common.cuh"
#include "gmg_impl.h"
#include "gridcomm.cuh"
#include "simpfem.h"

namespace simpfem {
namespace {

constexpr int kMaxOff = 343;  // offsets within radius <= 3.5 in a 7^3 box
constexpr int kSimpBlocks = 296, kSimpThreads = 256;

// Neighbours within the radius: a kernel argument, so that calls of different radii on
// other streams or from other threads do not meet.
struct FilterOffsets {
  double w[kMaxOff];
  int n;
  int8_t dx[kMaxOff], dy[kMaxOff], dz[kMaxOff];
};
static_assert(sizeof(FilterOffsets) <= 3900, "kernel arguments");

// y = H x (transpose = 0) or y = H^T x (transpose = 1); H symmetric in its
// weights, so (H^T x)_e = sum over neighbours f of w(e, f) x_f / rowsum_f.
//
// A block stages a tile of x with a halo of r = floor(rmin) elements in shared
// memory (zeros outside the grid, so the sum needs no bounds checks) and each
// thread forms kFilterPer outputs with independent accumulators.  A row sum
// depends only on how many elements lie within r on either side along each
// axis, so the block tabulates it once per combination that occurs (27 at r = 1)
// instead of once per element or, in H^T, once per neighbour: that scan of 19
// offsets inside a loop over 19 offsets (plus a division each) bound the
// element-per-thread kernel this replaces.  1M elements, rmin 1.5: 143 us -> 20.7 us
// (H and H^T alike; the 16 MB take 2.4 us, the 19 shared-memory reads an output
// are the larger part).
constexpr int kFilterThreads = 256, kFilterPer = 8;

struct FilterTile {
  int r;           // halo
  int tx, ty, tz;  // outputs per block: tx * ty * tz <= kFilterThreads * kFilterPer
  int bx, by, bz;  // blocks per axis
};

__device__ __forceinline__ int axis_code(int i, int n, int r) { return min(i, r) * (r + 1) + min(n - 1 - i, r); }

__global__ void __launch_bounds__(kFilterThreads) cone_filter_kernel(
    const __grid_constant__ FilterOffsets nb, int nx, int ny, int nz, FilterTile ft, int transpose,
    const double* __restrict__ x, double* __restrict__ y) {
  extern __shared__ __align__(16) double fsm[];
  const int r = ft.r, NC = (r + 1) * (r + 1), HY = ft.ty + 2 * r, HZ = ft.tz + 2 * r, HX = ft.tx + 2 * r;
  const int ntile = HX * HY * HZ;
  double* rs = fsm;                 // row sums by axis codes: [NC][NC][NC]
  double* tile = rs + NC * NC * NC;
  int* off = reinterpret_cast<int*>(tile + ntile);
  const int bz = blockIdx.x % ft.bz, bq = blockIdx.x / ft.bz, by = bq % ft.by, bx = bq / ft.by;
  const int i0 = bx * ft.tx, j0 = by * ft.ty, k0 = bz * ft.tz;
  for (int q = threadIdx.x; q < nb.n; q += kFilterThreads)
    off[q] = (nb.dx[q] * HY + nb.dy[q]) * HZ + nb.dz[q];
  for (int c = threadIdx.x; c < NC * NC * NC; c += kFilterThreads) {
    const int cz = c % NC, cy = (c / NC) % NC, cx = c / (NC * NC);
    const int xa = cx / (r + 1), xb = cx % (r + 1), ya = cy / (r + 1), yb = cy % (r + 1), za = cz / (r + 1),
              zb = cz % (r + 1);
    // elements within r on either side: both counts short only on an axis of at most 2r elements
    const bool occurs = (xa == r || xb == r || nx <= 2 * r) && (ya == r || yb == r || ny <= 2 * r) &&
                        (za == r || zb == r || nz <= 2 * r);
    double s = 0.0;
    if (occurs)
      for (int q = 0; q < nb.n; ++q) {
        const int dx = nb.dx[q], dy = nb.dy[q], dz = nb.dz[q];
        if (dx >= -xa && dx <= xb && dy >= -ya && dy <= yb && dz >= -za && dz <= zb) s += nb.w[q];
      }
    rs[c] = s;
  }
  if (transpose) __syncthreads();
  for (int t = threadIdx.x; t < ntile; t += kFilterThreads) {
    const int hz = t % HZ, hq = t / HZ, hy = hq % HY, hx = hq / HY;
    const int i = i0 + hx - r, j = j0 + hy - r, k = k0 + hz - r;
    double v = 0.0;
    if (i >= 0 && i < nx && j >= 0 && j < ny && k >= 0 && k < nz) {
      v = x[((int64_t)i * ny + j) * nz + k];
      if (transpose) v = v / rs[(axis_code(i, nx, r) * NC + axis_code(j, ny, r)) * NC + axis_code(k, nz, r)];
    }
    tile[t] = v;
  }
  __syncthreads();
  const int nout = ft.tx * ft.ty * ft.tz;
  int at[kFilterPer];
  double acc[kFilterPer];
#pragma unroll
  for (int m = 0; m < kFilterPer; ++m) {
    const int t = min((int)threadIdx.x + m * kFilterThreads, nout - 1);
    const int lz = t % ft.tz, lq = t / ft.tz, ly = lq % ft.ty, lx = lq / ft.ty;
    at[m] = ((lx + r) * HY + ly + r) * HZ + lz + r;
    acc[m] = 0.0;
  }
  for (int q = 0; q < nb.n; ++q) {
    const double w = nb.w[q];
    const int o = off[q];
#pragma unroll
    for (int m = 0; m < kFilterPer; ++m) acc[m] += w * tile[at[m] + o];
  }
#pragma unroll
  for (int m = 0; m < kFilterPer; ++m) {
    const int t = threadIdx.x + m * kFilterThreads;
    if (t >= nout) break;
    const int lz = t % ft.tz, lq = t / ft.tz, ly = lq % ft.ty, lx = lq / ft.ty;
    const int i = i0 + lx, j = j0 + ly, k = k0 + lz;
    if (i >= nx || j >= ny || k >= nz) continue;
    const int64_t e = ((int64_t)i * ny + j) * nz + k;
    y[e] = transpose ? acc[m]
                     : acc[m] / rs[(axis_code(i, nx, r) * NC + axis_code(j, ny, r)) * NC + axis_code(k, nz, r)];
  }
}

// A tile holds whole rows along z up to 64 elements (else 32, so that the halo
// stays a small share of a row) and is filled up along y and x to at most
// kFilterThreads * kFilterPer outputs with y about as long as x: the halo of a
// cube is the smallest.  On a rod, which is filled along x alone, the halo is a
// multiple of the outputs; there x is shortened until the tile fits.
constexpr size_t kFilterSmem = 227 * 1024;
size_t filter_smem(const FilterTile& f) {
  const size_t nc = (size_t)(f.r + 1) * (f.r + 1), h = 2 * f.r;
  return sizeof(double) * (nc * nc * nc + (f.tx + h) * (f.ty + h) * (f.tz + h)) + sizeof(int) * kMaxOff;
}

FilterTile filter_tile(int nx, int ny, int nz, int r) {
  FilterTile f;
  f.r = r;
  f.tz = nz <= 64 ? nz : 32;
  const int plane = std::max(1, kFilterThreads * kFilterPer / f.tz);
  int side = 1;
  while ((side + 1) * (side + 1) <= plane) ++side;
  f.ty = std::min(ny, side);
  f.tx = std::min(nx, std::max(1, plane / f.ty));
  while (f.tx > 1 && filter_smem(f) > kFilterSmem) f.tx = (f.tx + 1) / 2;
  f.bx = div_up(nx, f.tx);
  f.by = div_up(ny, f.ty);
  f.bz = div_up(nz, f.tz);
  return f;
}

cudaError_t launch_filter(const FilterOffsets& nb, int nx, int ny, int nz, int transpose, const double* x, double* y,
                          cudaStream_t s) {
  const FilterTile f = filter_tile(nx, ny, nz, (int)floor(nb.w[0]));  // the element's own weight is the radius
  const size_t smem = filter_smem(f);
  static std::atomic<uint64_t> attr_done;
  const cudaError_t e = once_per_device(attr_done, [] {
    return cudaFuncSetAttribute(cone_filter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFilterSmem);
  });
  if (e != cudaSuccess) return e;
  cone_filter_kernel<<<f.bx * f.by * f.bz, kFilterThreads, smem, s>>>(nb, nx, ny, nz, f, transpose, x, y);
  return sf_launched(1);
}

__device__ __forceinline__ double block_reduce_sum(double v, double* sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += sh[w];
  return t;
}

__device__ __forceinline__ double block_reduce_max(double v, double* sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t = fmax(t, sh[w]);
  return t;
}

// the reference's OC candidate for multiplier lm (simp_gpu.py:271-276):
// rn = clip(clip(rho * sqrt(-dc_s / (lm * dv_s)), rho - move, rho + move), 1e-3, 1)
// with dc_s = min(dc, -1e-12), dv_s = max(dv, 1e-12)
__device__ __forceinline__ double oc_candidate(double rho, double dc, double dv, double lm, double move) {
  const double dcs = fmin(dc, -1e-12), dvs = fmax(dv, 1e-12);
  double r = rho * sqrt(-dcs / (lm * dvs));
  r = fmin(fmax(r, rho - move), rho + move);
  return fmin(fmax(r, 1e-3), 1.0);
}

// partial sums of vw rn(lm): the volume of a candidate, a launch per bisection step
__global__ void __launch_bounds__(kSimpThreads) oc_volume_kernel(int64_t n, const double* __restrict__ rho,
                                                                 const double* __restrict__ dc,
                                                                 const double* __restrict__ dv,
                                                                 const double* __restrict__ vw, double lm, double move,
                                                                 double* __restrict__ partials) {
  __shared__ double sh[32];
  double v = 0.0;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x)
    v += vw[e] * oc_candidate(rho[e], dc[e], dv ? dv[e] : 1.0, lm, move);
  const double t = block_reduce_sum(v, sh);
  if (threadIdx.x == 0) partials[blockIdx.x] = t;
}

// rn(lm) and partial maxima of |rn - rho|
__global__ void __launch_bounds__(kSimpThreads) oc_candidate_kernel(int64_t n, const double* __restrict__ rho,
                                                                    const double* __restrict__ dc,
                                                                    const double* __restrict__ dv, double lm,
                                                                    double move, double* __restrict__ rn,
                                                                    double* __restrict__ partials) {
  __shared__ double sh[32];
  double v = 0.0;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    const double r = oc_candidate(rho[e], dc[e], dv ? dv[e] : 1.0, lm, move);
    rn[e] = r;
    v = fmax(v, fabs(r - rho[e]));
  }
  const double t = block_reduce_max(v, sh);
  if (threadIdx.x == 0) partials[blockIdx.x] = t;
}

// out = the partials summed (max = 0) or maximised (max = 1) by one block in a
// fixed order
__global__ void __launch_bounds__(kSimpThreads) oc_finish_kernel(int nb, int max, const double* __restrict__ partials,
                                                                 double* __restrict__ out) {
  __shared__ double sh[32];
  double s = 0.0;
  for (int b = threadIdx.x; b < nb; b += kSimpThreads) s = max ? fmax(s, partials[b]) : s + partials[b];
  const double t = max ? block_reduce_max(s, sh) : block_reduce_sum(s, sh);
  if (threadIdx.x == 0) *out = t;
}

// Heaviside projection of x and its derivative (pub_simp_solver.py:245-253):
// p = (tanh(b eta) + tanh(b (x - eta))) / den, dp = b (1 - tanh(b (x - eta))^2) / den,
// den = tanh(b eta) + tanh(b (1 - eta)); dc (optional) is multiplied by dp into dcdp.
__global__ void heaviside_kernel(int64_t n, const double* __restrict__ x, double beta, double eta, double tbe,
                                 double den, double* __restrict__ p, double* __restrict__ dp,
                                 const double* __restrict__ dc, double* __restrict__ dcdp) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  const double t = tanh(beta * (x[e] - eta));
  if (p) p[e] = (tbe + t) / den;
  const double d = beta * (1.0 - t * t) / den;
  if (dp) dp[e] = d;
  if (dcdp) dcdp[e] = dc[e] * d;
}

// partial sums of tanh(b eta) + tanh(b (x - eta)) (the projected volume times den)
__global__ void __launch_bounds__(kSimpThreads) projected_sum_kernel(int64_t n, const double* __restrict__ x,
                                                                     double beta, double eta, double tbe,
                                                                     double* __restrict__ partials) {
  __shared__ double sh[32];
  double v = 0.0;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x)
    v += tbe + tanh(beta * (x[e] - eta));
  const double t = block_reduce_sum(v, sh);
  if (threadIdx.x == 0) partials[blockIdx.x] = t;
}

// The whole OC bisection in one cooperative launch.
//
// The volume of a candidate is a sum over all elements, so one bisection step is
// a pass over the design and a grid-wide sum; launched step by step it cost 37 us
// at 1M elements (pass 7.4, one-thread finish 6.6, copy, host decision), sixty
// times over.  Here each block keeps its elements' four numbers in shared memory
// (A = rho sqrt(-dc / dv), the two bounds and vw: 216 KB a block at 1M elements; elements
// beyond the capacity are formed again from global memory in every pass), the
// candidate for multiplier lm is clip(A / sqrt(lm)), and every block takes the
// bisection's decisions itself from the same sums.  A pass evaluates the midpoint
// and both midpoints that can follow it, so two steps of the sequential bisection
// share one exchange (its latency, not the arithmetic, is the larger part).  The
// update itself is evaluated with the reference's expression.  1M elements:
// 2.2 ms -> 143 us for the 60 steps.
constexpr int kOcThreads = 512;

// clip(A q, lo, hi) by comparisons (fmin / fmax add NaN handling on the FP64
// pipe); a NaN A q takes lo, as fmax does
__device__ __forceinline__ double oc_clip(double t, double lo, double hi) {
  t = t > lo ? t : lo;
  return t < hi ? t : hi;
}
__device__ __forceinline__ void oc_bounds(double rho, double move, double& lo, double& hi) {
  lo = fmin(fmax(rho - move, 1e-3), 1.0);
  hi = fmin(fmax(rho + move, 1e-3), 1.0);
}

__global__ void __launch_bounds__(kOcThreads, 1)
    oc_bisect_kernel(int64_t n, const double* __restrict__ rho, const double* __restrict__ dc,
                     const double* __restrict__ dv, const double* __restrict__ vw, double target, double move,
                     int keep, double* rn, GridExchange x, double* __restrict__ out) {
  extern __shared__ __align__(16) double osm[];  // [4][keep][kOcThreads]
  __shared__ double red[3][kOcThreads / 32];
  __shared__ double sums[3];
  __shared__ int good;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int64_t stride = (int64_t)gridDim.x * kOcThreads, first = (int64_t)blockIdx.x * kOcThreads + tid;
  double* sA = osm;
  double* sL = sA + (size_t)keep * kOcThreads;
  double* sH = sL + (size_t)keep * kOcThreads;
  double* sV = sH + (size_t)keep * kOcThreads;
  auto scale = [&](int64_t e, double r) {
    const double dcs = fmin(dc[e], -1e-12), dvs = fmax(dv ? dv[e] : 1.0, 1e-12);
    return r * sqrt(-dcs / dvs);
  };
  for (int k = 0; k < keep; ++k) {
    const int64_t e = first + k * stride;
    double A = 0.0, lo = 0.0, hi = 0.0, v = 0.0;
    if (e < n) {
      const double r = rho[e];
      A = scale(e, r);
      oc_bounds(r, move, lo, hi);
      v = vw[e];
    }
    sA[k * kOcThreads + tid] = A;
    sL[k * kOcThreads + tid] = lo;
    sH[k * kOcThreads + tid] = hi;
    sV[k * kOcThreads + tid] = v;
  }
  unsigned epoch = 0;
  double l1 = 0.0, l2 = 1e9, lm = 0.5 * (l1 + l2);
  int steps = 0;
  bool ok = true;
  // the reference's bisection (simp_gpu.py:268-290): at most 100 steps, stop when l2 - l1 < 1e-9
  while (steps < 100) {
    const double m = 0.5 * (l1 + l2);
    const double qa = 1.0 / sqrt(m), qb = 1.0 / sqrt(0.5 * (l1 + m)), qc = 1.0 / sqrt(0.5 * (m + l2));
    double v[3] = {0.0, 0.0, 0.0};
    for (int k = 0; k < keep; ++k) {
      const double A = sA[k * kOcThreads + tid], w = sV[k * kOcThreads + tid];
      const double lo = sL[k * kOcThreads + tid], hi = sH[k * kOcThreads + tid];
      v[0] += w * oc_clip(A * qa, lo, hi);
      v[1] += w * oc_clip(A * qb, lo, hi);
      v[2] += w * oc_clip(A * qc, lo, hi);
    }
    for (int64_t e = first + keep * stride; e < n; e += stride) {
      const double r = rho[e], A = scale(e, r), w = vw[e];
      double lo, hi;
      oc_bounds(r, move, lo, hi);
      v[0] += w * oc_clip(A * qa, lo, hi);
      v[1] += w * oc_clip(A * qb, lo, hi);
      v[2] += w * oc_clip(A * qc, lo, hi);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v[c] += __shfl_down_sync(0xffffffffu, v[c], o);
      if (lane == 0) red[c][wid] = v[c];
    }
    __syncthreads();
    ++epoch;
    if (wid == 0) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        v[c] = lane < kOcThreads / 32 ? red[c][lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[c] += __shfl_down_sync(0xffffffffu, v[c], o);
      }
      const bool all = grid_allreduce_warp<3>(x, epoch, v);
      if (lane == 0) {
        sums[0] = v[0];
        sums[1] = v[1];
        sums[2] = v[2];
        good = all ? 1 : 0;
      }
    }
    __syncthreads();
    ok = good != 0;
    if (!ok) break;
    // step one at m, then step two at the midpoint that follows from it
    lm = m;
    ++steps;
    const bool high = sums[0] > target;
    if (high) l1 = lm;
    else l2 = lm;
    if (l2 - l1 < 1e-9 || steps >= 100) break;
    lm = 0.5 * (l1 + l2);
    ++steps;
    if (sums[high ? 2 : 1] > target) l1 = lm;
    else l2 = lm;
    if (l2 - l1 < 1e-9) break;
  }
  double ch[1] = {0.0};
  if (ok)
    for (int64_t e = first; e < n; e += stride) {
      const double r = rho[e], c = oc_candidate(r, dc[e], dv ? dv[e] : 1.0, lm, move);
      ch[0] = fmax(ch[0], fabs(c - r));
      rn[e] = c;
    }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ch[0] = fmax(ch[0], __shfl_down_sync(0xffffffffu, ch[0], o));
  if (lane == 0) red[0][wid] = ch[0];
  __syncthreads();
  if (wid == 0 && ok) {
    ch[0] = lane < kOcThreads / 32 ? red[0][lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ch[0] = fmax(ch[0], __shfl_down_sync(0xffffffffu, ch[0], o));
    ok = grid_allreduce_warp<1, true>(x, epoch + 1, ch);
  }
  if (blockIdx.x == 0 && tid == 0) {
    out[0] = ch[0];
    out[1] = lm;
    out[2] = (double)steps;
    out[3] = ok ? 0.0 : 1.0;
  }
}

FilterOffsets make_offsets(double rmin) {
  FilterOffsets o{};
  const int r = (int)floor(rmin);
  o.n = 0;
  // the element itself first, weight rmin, then the other offsets in
  // lexicographic order, weight rmin - dist (kept when dist <= rmin - 1e-10)
  o.dx[0] = o.dy[0] = o.dz[0] = 0;
  o.w[0] = rmin;
  o.n = 1;
  for (int a = -r; a <= r; ++a)
    for (int b = -r; b <= r; ++b)
      for (int c = -r; c <= r; ++c) {
        if (a == 0 && b == 0 && c == 0) continue;
        const double d = sqrt((double)(a * a + b * b + c * c));
        if (d > rmin - 1e-10) continue;
        o.dx[o.n] = (int8_t)a;
        o.dy[o.n] = (int8_t)b;
        o.dz[o.n] = (int8_t)c;
        o.w[o.n] = rmin - d;
        ++o.n;
      }
  return o;
}

}  // namespace
}  // namespace simpfem

using namespace simpfem;

#define SIMP_API_BEGIN try {
#define SIMP_API_END                        \
  }                                         \
  catch (const CudaFailure&) {              \
    return SIMPFEM_ECUDA;                   \
  }                                         \
  catch (const InvalidArg& e) {             \
    set_error(e.msg);                       \
    return SIMPFEM_EINVAL;                  \
  }                                         \
  catch (const std::exception& e) {         \
    set_error(e.what());                    \
    return SIMPFEM_EINTERNAL;               \
  }                                         \
  return SIMPFEM_OK;

extern "C" {

int simpfem_cone_filter(int nx, int ny, int nz, double rmin, int transpose, const double* x, double* y,
                        void* stream) {
  SIMP_API_BEGIN
  if (nx < 1 || ny < 1 || nz < 1 || !x || !y || x == y) throw InvalidArg{"simpfem_cone_filter: bad argument"};
  if (!(rmin >= 1.0 && rmin <= 3.5)) throw InvalidArg{"simpfem_cone_filter: rmin must be in [1, 3.5]"};
  cudaStream_t s = (cudaStream_t)stream;
  SF_CUDA(launch_filter(make_offsets(rmin), nx, ny, nz, transpose ? 1 : 0, x, y, s));
  SIMP_API_END
}

// the exchange slots, the four results, and room to start the slots on 16 bytes
size_t simpfem_oc_work_bytes(void) { return kGridCommBytes + sizeof(double) * 4 + 8; }

// The bisection by a launch and a synchronisation per step, for devices that cannot hold
// the grid of the one launch: h = {change, lm, steps}.
static void oc_bisect_launched(int64_t n, const double* rho, const double* dc, const double* dv, const double* vol_w,
                               double target, double move, double* rho_new, double* partials, double* out,
                               cudaStream_t s, double (&h)[4]) {
  const int nb = (int)std::min<int64_t>(kSimpBlocks, div_up(n, kSimpThreads));
  auto finish = [&](int max) {
    oc_finish_kernel<<<1, kSimpThreads, 0, s>>>(nb, max, partials, out);
    SF_CUDA(sf_launched(2));
    double v = 0.0;
    SF_CUDA(cudaMemcpyAsync(&v, out, sizeof(v), cudaMemcpyDeviceToHost, s));
    SF_CUDA(cudaStreamSynchronize(s));
    return v;
  };
  double l1 = 0.0, l2 = 1e9, lm = 0.5 * (l1 + l2);
  int steps = 0;
  for (int it = 0; it < 100; ++it) {
    lm = 0.5 * (l1 + l2);
    oc_volume_kernel<<<nb, kSimpThreads, 0, s>>>(n, rho, dc, dv, vol_w, lm, move, partials);
    const double vol = finish(0);
    ++steps;
    if (vol > target) l1 = lm;
    else l2 = lm;
    if (l2 - l1 < 1e-9) break;
  }
  oc_candidate_kernel<<<nb, kSimpThreads, 0, s>>>(n, rho, dc, dv, lm, move, rho_new, partials);
  h[0] = finish(1);
  h[1] = lm;
  h[2] = steps;
  h[3] = 0.0;
}

// blocks of the one-launch bisection that the device holds at once
static int oc_coresident() {
  constexpr int kMost = 224 * 1024;
  static std::atomic<int> cached[64];  // 0 unknown, else the number + 1
  int dev = 0;
  SF_CUDA(cudaGetDevice(&dev));
  int v = dev < 64 ? cached[dev].load(std::memory_order_relaxed) : 0;
  if (v == 0) {
    SF_CUDA(cudaFuncSetAttribute(oc_bisect_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMost));
    v = grid_coresident((const void*)oc_bisect_kernel, kOcThreads, kMost) + 1;
    if (dev < 64) cached[dev].store(v, std::memory_order_relaxed);
  }
  return v - 1;
}

static int oc_update(int64_t n, const double* rho, const double* dc, const double* dv, const double* vol_w,
                     double volfrac, double move, double* rho_new, double* work, size_t work_bytes,
                     double* change_host, double* lambda_host, int* steps_host, const GridWait& wait, void* stream) {
  SIMP_API_BEGIN
  if (n < 1 || !rho || !dc || !vol_w || !rho_new || !work) throw InvalidArg{"simpfem_oc_update: null argument"};
  if (work_bytes < simpfem_oc_work_bytes()) throw InvalidArg{"simpfem_oc_update: workspace too small"};
  cudaStream_t s = (cudaStream_t)stream;
  // the slots are read and written as pairs of words; work is aligned to its type only
  GridExchange x;
  x.slots = (ulonglong2*)(((uintptr_t)work + 15) / 16 * 16);
  x.polls = wait.polls;
  x.polls0 = wait.polls0;
  static_assert(kGridCommBytes >= sizeof(double) * kSimpBlocks, "partial sums of the launched form");
  double* out = (double*)x.slots + kGridCommBytes / sizeof(double);
  double target = volfrac * (double)n, h[4];
  const int most = wait.one_launch ? oc_coresident() : 0;
  bool done = false;
  if (most > 0) {
    // two elements a thread or more before another block joins (an exchange costs more the more blocks take part)
    const int nb = (int)std::min<int64_t>(std::min(most, grid_sm_count()), div_up(n, 2 * kOcThreads));
    constexpr int kMaxKeep = 224 * 1024 / (4 * 8 * kOcThreads);
    int keep = (int)std::min<int64_t>(kMaxKeep, div_up(n, (int64_t)nb * kOcThreads));
    SF_CUDA(cudaMemsetAsync(x.slots, 0, kGridCommBytes, s));
    void* args[] = {&n,      (void*)&rho, (void*)&dc, (void*)&dv, (void*)&vol_w, &target,
                    &move,   &keep,       &rho_new,   &x,         &out};
    const cudaError_t e = cudaLaunchCooperativeKernel((const void*)oc_bisect_kernel, dim3(nb), dim3(kOcThreads), args,
                                                      sizeof(double) * 4 * (size_t)keep * kOcThreads, s);
    done = !grid_refused(e);
    if (done) {
      SF_CUDA(e);
      SF_CUDA(sf_launched(1));
      SF_CUDA(cudaMemcpyAsync(h, out, sizeof(h), cudaMemcpyDeviceToHost, s));
      SF_CUDA(cudaStreamSynchronize(s));
      if (h[3] != 0.0) throw std::runtime_error("simpfem_oc_update: a grid exchange ran out of its wait");
    }
  }
  if (!done) oc_bisect_launched(n, rho, dc, dv, vol_w, target, move, rho_new, (double*)x.slots, out, s, h);
  if (change_host) *change_host = h[0];
  if (lambda_host) *lambda_host = h[1];
  if (steps_host) *steps_host = (int)h[2];
  SIMP_API_END
}

int simpfem_oc_update(int64_t n, const double* rho, const double* dc, const double* dv, const double* vol_w,
                      double volfrac, double move, double* rho_new, double* work, size_t work_bytes,
                      double* change_host, double* lambda_host, int* steps_host, void* stream) {
  return oc_update(n, rho, dc, dv, vol_w, volfrac, move, rho_new, work, work_bytes, change_host, lambda_host,
                   steps_host, GridWait(), stream);
}

void simpfem_oc_update_opts(int64_t n, const double* rho, const double* dc, const double* dv, const double* vol_w,
                            double volfrac, double move, double* rho_new, double* work, size_t work_bytes,
                            double* change_host, double* lambda_host, int* steps_host,
                            const simpfem_grid_opts* opts, void* stream, int* status) {
  const int st = oc_update(n, rho, dc, dv, vol_w, volfrac, move, rho_new, work, work_bytes, change_host, lambda_host,
                           steps_host, grid_wait(opts), stream);
  if (status) *status = st;
}

int simpfem_heaviside(int64_t n, const double* x, double beta, double eta, double* proj, double* dproj,
                      void* stream) {
  SIMP_API_BEGIN
  if (n < 1 || !x || (!proj && !dproj)) throw InvalidArg{"simpfem_heaviside: bad argument"};
  if (!(beta > 0.0)) throw InvalidArg{"simpfem_heaviside: beta must be positive"};
  const double tbe = tanh(beta * eta), den = tbe + tanh(beta * (1.0 - eta));
  cudaStream_t s = (cudaStream_t)stream;
  heaviside_kernel<<<div_up(n, 256), 256, 0, s>>>(n, x, beta, eta, tbe, den, proj, dproj, nullptr, nullptr);
  SF_CUDA(sf_launched(1));
  SIMP_API_END
}

size_t simpfem_oc_projected_work_bytes(int64_t n) {
  return sizeof(double) * (5 * (size_t)std::max<int64_t>(n, 1) + kSimpBlocks + 2);
}

int simpfem_oc_update_projected(int nx, int ny, int nz, double rmin, const double* rho, const double* rho_f,
                                const double* dc_phys, double beta, double eta, double volfrac, double move,
                                double* rho_new, double* work, size_t work_bytes, double* change_host,
                                double* lambda_host, int* steps_host, void* stream) {
  SIMP_API_BEGIN
  const int64_t n = (int64_t)nx * ny * nz;
  if (nx < 1 || ny < 1 || nz < 1 || !rho || !rho_f || !dc_phys || !rho_new || !work)
    throw InvalidArg{"simpfem_oc_update_projected: null argument"};
  if (work_bytes < simpfem_oc_projected_work_bytes(n))
    throw InvalidArg{"simpfem_oc_update_projected: workspace too small"};
  if (!(beta > 1e-6)) throw InvalidArg{"simpfem_oc_update_projected: beta must exceed 1e-6 (else simpfem_oc_update)"};
  if (!(rmin >= 1.0 && rmin <= 3.5)) throw InvalidArg{"simpfem_oc_update_projected: rmin must be in [1, 3.5]"};
  cudaStream_t s = (cudaStream_t)stream;
  const FilterOffsets around = make_offsets(rmin);
  double* dh = work;
  double* dcdh = dh + n;  // dc * dh, then reused for the filtered candidate
  double* dcd = dcdh + n;
  double* dvd = dcd + n;
  double* rn = dvd + n;
  double* partials = rn + n;
  double* out = partials + kSimpBlocks;
  const double tbe = tanh(beta * eta), den = tbe + tanh(beta * (1.0 - eta));
  const int eb = div_up(n, 256);
  // sensitivities in the design space (simp_gpu.py:245-258): H^T (dc dh), H^T dh
  heaviside_kernel<<<eb, 256, 0, s>>>(n, rho_f, beta, eta, tbe, den, nullptr, dh, dc_phys, dcdh);
  SF_CUDA(sf_launched(1));
  SF_CUDA(launch_filter(around, nx, ny, nz, 1, dcdh, dcd, s));
  SF_CUDA(launch_filter(around, nx, ny, nz, 1, dh, dvd, s));
  double* rnf = dcdh;
  const int nb = (int)std::min<int64_t>(kSimpBlocks, div_up(n, kSimpThreads));
  const double target = volfrac * (double)n;
  double l1 = 0.0, l2 = 1e9, lm = 0.5 * (l1 + l2);
  int steps = 0;
  // the bisection of simp_gpu.py:268-290 with the projected volume of each candidate:
  // sum(tanh(b eta) + tanh(b (H rn - eta))) / den against volfrac n
  for (int it = 0; it < 100; ++it) {
    lm = 0.5 * (l1 + l2);
    oc_candidate_kernel<<<nb, kSimpThreads, 0, s>>>(n, rho, dcd, dvd, lm, move, rn, partials);
    SF_CUDA(launch_filter(around, nx, ny, nz, 0, rn, rnf, s));
    projected_sum_kernel<<<nb, kSimpThreads, 0, s>>>(n, rnf, beta, eta, tbe, partials);
    oc_finish_kernel<<<1, kSimpThreads, 0, s>>>(nb, 0, partials, out);
    SF_CUDA(sf_launched(3));
    double vol = 0.0;
    SF_CUDA(cudaMemcpyAsync(&vol, out, sizeof(double), cudaMemcpyDeviceToHost, s));
    SF_CUDA(cudaStreamSynchronize(s));
    ++steps;
    if (vol / den > target) l1 = lm;
    else l2 = lm;
    if (l2 - l1 < 1e-9) break;
  }
  oc_candidate_kernel<<<nb, kSimpThreads, 0, s>>>(n, rho, dcd, dvd, lm, move, rho_new, partials);
  oc_finish_kernel<<<1, kSimpThreads, 0, s>>>(nb, 1, partials, out);
  SF_CUDA(sf_launched(2));
  double ch = 0.0;
  SF_CUDA(cudaMemcpyAsync(&ch, out, sizeof(double), cudaMemcpyDeviceToHost, s));
  SF_CUDA(cudaStreamSynchronize(s));
  if (change_host) *change_host = ch;
  if (lambda_host) *lambda_host = lm;
  if (steps_host) *steps_host = steps;
  SIMP_API_END
}

}  // extern "C"
