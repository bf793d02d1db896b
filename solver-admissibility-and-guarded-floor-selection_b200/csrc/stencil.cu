// Coarse-level operators of the Galerkin hierarchy as 27-point 3x3-block stencils.
//
// The reference assembles level 1 elementwise into CSR
// (gpu_fem/multigrid_v4.py:219-361, _build_level1_galerkin_struct +
// assemble_level1_galerkin) and forms level >= 2 with sparse triple products
// (gpu_fem/multigrid_v4.py:1275-1300); transfers are CSR SpMVs with
// kron(P_scalar, I3) restricted to free DOFs (gpu_fem/solver_v2.py:62-149,
// multigrid_v4.py:728-748).  On the structured grid every one of these is a
// stencil: the coarse operator of node n is 27 blocks of 3x3 coupling n to its
// neighbours n + o, and the trilinear transfers are separable products of 1-D
// weights.  Coefficients are stored structure-of-arrays,
// coef[(o * 9 + r * 3 + q) * nn + n], so a warp of consecutive nodes reads each
// coefficient with one coalesced access.
#include "common.cuh"

namespace simpfem {

__device__ __forceinline__ void node_ijk(const Grid& g, int64_t node, int& i, int& j, int& k) {
  const int NZ = g.nz + 1, NY = g.ny + 1;
  k = (int)(node % NZ);
  j = (int)((node / NZ) % NY);
  i = (int)(node / ((int64_t)NZ * NY));
}

__device__ __forceinline__ int64_t node_id(const Grid& g, int i, int j, int k) {
  return ((int64_t)i * (g.ny + 1) + j) * (g.nz + 1) + k;
}

// Unsigned division by an invariant d >= 1 for dividends below 2^31: one multiply
// instead of the twenty instructions of an integer division (Granlund and Montgomery,
// "Division by invariant integers using multiplication", 1994, figure 4.1).
struct FastDiv {
  unsigned d = 1, mul = 0, shift = 0;
  static FastDiv make(unsigned d) {
    FastDiv f;
    f.d = d;
    unsigned l = 0;
    while ((1u << l) < d && l < 31) ++l;  // 2^l >= d
    f.shift = l;
    f.mul = (unsigned)((((uint64_t)1 << 32) * (((uint64_t)1 << l) - d)) / d + 1);
    return f;
  }
  __device__ __forceinline__ unsigned div(unsigned n) const {
    return (unsigned)(((uint64_t)__umulhi(n, mul) + n) >> shift);
  }
};
// node_ijk by multiplications; dz, dy divide by nz + 1 and ny + 1
__device__ __forceinline__ void node_ijk(const Grid& g, const FastDiv& dz, const FastDiv& dy, int n, int& i, int& j,
                                         int& k) {
  const int jq = (int)dz.div(n);
  k = n - jq * (g.nz + 1);
  i = (int)dy.div(jq);
  j = jq - i * (g.ny + 1);
}

// 32 nodes a block, nine warps: warp col = 3 ox + oy loads what couples its 32 nodes'
// rows to their three z-neighbours in column (ox, oy) -- 27 coefficients and nine
// vector entries a lane, coalesced over the nodes and all in flight together -- and
// the warps then take up the rows' sums one after the other, column by column, so
// a row is one chain of 81 multiply-adds in the operator's order (nested Krylov
// solves hang on its last bit); 96 threads apply the epilogue with operands they read
// up front.  (A thread per row had 6 warps on an SM for its 81 loads: 8.0 us on the
// 9,471 + 1,386 nodes of the two coarse levels of 80 x 40 x 20, now 3.9; reading the
// operator from L2 takes 2.  69,741 nodes are bound by their 136 MB of coefficients
// either way.)  A neighbour outside the grid has zero coefficients (the
// assembly writes them), so its offset is clamped to 0 instead of branching.  32-bit
// node indices (levels >= 1 have at most 1/8 of the fine nodes; the launcher checks
// 3 * nn < 2^31).
constexpr int kStencilNodes = 32, kStencilThreads = 9 * 32;

template <typename VT, int EPI>
__global__ void __launch_bounds__(kStencilThreads) stencil_kernel(Grid g, FastDiv dz, FastDiv dy,
                                                                  const VT* __restrict__ coef,
                                                                  const uint8_t* __restrict__ mask,
                                                                  const VT* __restrict__ u, EpiArgs ea) {
  if (guard_off(ea.guard)) return;
  __shared__ VT part[kStencilNodes * 3];
  const int nn = (int)g.nn, tid = threadIdx.x, col = tid >> 5, nl = tid & 31;
  const int n0 = blockIdx.x * kStencilNodes, n = min(n0 + nl, nn - 1);
  const int dof = 3 * n0 + tid;
  const bool row = tid < 3 * kStencilNodes && dof < 3 * nn;
  VT ob = VT(0), od = VT(0), oi = VT(0), ox_ = VT(0);
  uint8_t fr = 0;
  if (row) {
    fr = mask[dof];
    if (EPI != EPI_APPLY) ob = ((const VT*)ea.b)[dof];
    if (EPI == EPI_CHEB1 || EPI == EPI_CHEB || EPI == EPI_JAC) oi = ((const VT*)ea.dinv)[dof];
    if (EPI == EPI_CHEB) od = ((const VT*)ea.d)[dof];
    if (EPI == EPI_CHEB1 || EPI == EPI_CHEB || EPI == EPI_JAC) ox_ = u[dof];
  }
  const int NZ1 = g.nz + 1, NY1 = g.ny + 1;
  const int jq = (int)dz.div(n), k = n - jq * NZ1, i = (int)dy.div(jq), j = jq - i * NY1;
  const int ox = col / 3, oy = col - 3 * ox;
  const int sx = ox == 0 ? (i > 0 ? -NY1 * NZ1 : 0) : (ox == 2 ? (i < g.nx ? NY1 * NZ1 : 0) : 0);
  const int sy = oy == 0 ? (j > 0 ? -NZ1 : 0) : (oy == 2 ? (j < g.ny ? NZ1 : 0) : 0);
  const VT* cp = coef + (int64_t)(col * 27) * nn + n;
  VT cf[27];
#pragma unroll
  for (int e = 0; e < 27; ++e) cf[e] = cp[(int64_t)e * nn];
  VT uv[9];
#pragma unroll
  for (int oz = 0; oz < 3; ++oz) {
    const int sz = oz == 0 ? (k > 0 ? -1 : 0) : (oz == 2 ? (k < g.nz ? 1 : 0) : 0);
    const VT* um = u + 3 * (n + sx + sy + sz);
#pragma unroll
    for (int q = 0; q < 3; ++q) uv[3 * oz + q] = um[q];
  }
  for (int c = 0; c < 9; ++c) {
    if (col == c) {
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        VT acc = c > 0 ? part[3 * nl + r] : VT(0);
#pragma unroll
        for (int e = 0; e < 9; ++e) acc = fma(cf[e / 3 * 9 + r * 3 + e % 3], uv[e], acc);
        part[3 * nl + r] = acc;
      }
    }
    __syncthreads();
  }
  if (!row) return;
  const VT ku = part[tid];
  const bool f = fr != 0;
  VT* py = (EPI == EPI_APPLY || EPI == EPI_RESID ? (VT*)ea.y : (VT*)ea.xo) + dof;
  VT res = VT(0), dn = VT(0);
  if (EPI == EPI_APPLY) {
    res = ku;
  } else if (EPI == EPI_RESID) {
    res = sub_rn(ob, ku);
  } else if (EPI == EPI_CHEB1) {
    dn = mul_rn(oi, sub_rn(ob, ku));
    res = add_rn(ox_, mul_rn((VT)ea.s1, dn));
  } else if (EPI == EPI_CHEB) {
    dn = mul_rn((VT)ea.s1, add_rn(mul_rn(oi, sub_rn(ob, ku)), mul_rn((VT)ea.s2, od)));
    res = add_rn(ox_, dn);
  } else {
    res = add_rn(ox_, mul_rn(mul_rn((VT)ea.s1, oi), sub_rn(ob, ku)));
  }
  *py = f ? res : VT(0);
  if (EPI == EPI_CHEB1 || EPI == EPI_CHEB) ((VT*)ea.d)[dof] = f ? dn : VT(0);
}

template <typename VT>
static cudaError_t stencil_dispatch(Epi epi, const Grid& g, const void* coef, const uint8_t* mask,
                                    const void* u, const EpiArgs& ea, cudaStream_t s) {
  if (3 * g.nn >= (int64_t(1) << 31)) return cudaErrorInvalidValue;
  const int bs = kStencilThreads, nb = div_up(g.nn, kStencilNodes);
  const FastDiv dz = FastDiv::make(g.nz + 1), dy = FastDiv::make(g.ny + 1);
  const VT* c = (const VT*)coef;
  const VT* uu = (const VT*)u;
  switch (epi) {
    case EPI_APPLY: stencil_kernel<VT, EPI_APPLY><<<nb, bs, 0, s>>>(g, dz, dy, c, mask, uu, ea); break;
    case EPI_RESID: stencil_kernel<VT, EPI_RESID><<<nb, bs, 0, s>>>(g, dz, dy, c, mask, uu, ea); break;
    case EPI_CHEB1: stencil_kernel<VT, EPI_CHEB1><<<nb, bs, 0, s>>>(g, dz, dy, c, mask, uu, ea); break;
    case EPI_CHEB: stencil_kernel<VT, EPI_CHEB><<<nb, bs, 0, s>>>(g, dz, dy, c, mask, uu, ea); break;
    case EPI_JAC: stencil_kernel<VT, EPI_JAC><<<nb, bs, 0, s>>>(g, dz, dy, c, mask, uu, ea); break;
    default: return cudaErrorInvalidValue;
  }
  return sf_launched(1);
}

cudaError_t launch_stencil(DType t, Epi epi, const Grid& g, const void* coef, const uint8_t* mask, const void* u,
                           const EpiArgs& ea, cudaStream_t s) {
  if (t == F64) return stencil_dispatch<double>(epi, g, coef, mask, u, ea, s);
  if (t == F32) return stencil_dispatch<float>(epi, g, coef, mask, u, ea, s);
  return cudaErrorInvalidValue;
}

// ----------------------------------------------------------------------------
// BF16 stencils of the mixed-precision cycle, by node and neighbour column.  The 27
// coefficients coupling node n to its three z-neighbours in column (ox, oy) are 32
// entries [oz * 9 + r * 3 + q] (27..31 zero), i.e. four 16-byte quarters; quarter q of
// the nine columns of three consecutive nodes is contiguous:
// coefC[((n / 3 * 4 + q) * 27 + n % 3 * 9 + col) * 8 + entry % 8], col = ox * 3 + oy.
// Made from the FP64 structure-of-arrays operator once per setup.
//
// Nine lanes per node, three nodes per warp: lane (t, col) loads its four quarters
// (a warp's 27 quarters are one run of 432 bytes) and the 9 vector entries of its
// z-neighbours and forms its part of the node's three row sums; nine lanes then add
// a row's nine parts each, in column order, and apply its epilogue.  The kernel is
// bound by its instructions (8.4 M at 69,741 nodes before, 361 a warp): the node's
// position comes from multiplications instead of divisions, and nine lanes instead of
// three share the sums (160 x 80 x 40, mean of its two smoothed levels: 9.0 us before,
// 6.1; 200 x 100 x 50: 15.4, 10.7; reading the larger level takes 6.1 and 12).
constexpr int kColSlot = 32, kNodeStrideC = 9 * kColSlot, kPackNodes = 30;

__device__ __forceinline__ int64_t col_slot(int n, int col, int quarter) {
  return ((int64_t)(n / 3 * 4 + quarter) * 27 + n % 3 * 9 + col) * 8;
}

// 30 nodes per block: coalesced reads along n of the FP64 operator, rounded into
// shared memory, 16-byte writes of the quarters
__global__ void __launch_bounds__(256) stencil_colmajor_bf16_kernel(int nn, const double* __restrict__ K64,
                                                                     __nv_bfloat16* __restrict__ out) {
  __shared__ __align__(16) __nv_bfloat16 tile[kPackNodes * kNodeStrideC];
  const int n0 = blockIdx.x * kPackNodes;
  const int nl = threadIdx.x & 31, c0 = threadIdx.x >> 5;
  const int cnt = min(kPackNodes, nn - n0);
  if (nl < kPackNodes)
    for (int c = c0; c < kNodeStrideC; c += 8) {
      const int col = c / kColSlot, w = c % kColSlot;
      float v = 0.f;
      if (nl < cnt && w < 27) {
        const int o = col * 3 + w / 9;  // o = ox * 9 + oy * 3 + oz
        v = (float)K64[(int64_t)(o * 9 + w % 9) * nn + n0 + nl];
      }
      tile[nl * kNodeStrideC + c] = __float2bfloat16_rn(v);
    }
  __syncthreads();
  // nodes beyond the last fill its group of three with zeros
  const int groups = (cnt + 2) / 3;
  for (int e = threadIdx.x; e < groups * 3 * 36; e += blockDim.x) {
    const int nd = e / 36, qc = e % 36, col = qc >> 2, q = qc & 3;
    *reinterpret_cast<uint4*>(out + col_slot(n0 + nd, col, q)) =
        *reinterpret_cast<const uint4*>(tile + nd * kNodeStrideC + col * kColSlot + q * 8);
  }
}

size_t stencil_colmajor_bytes(int64_t nn) { return (size_t)((nn + 2) / 3 * 3) * kNodeStrideC * 2; }

cudaError_t launch_stencil_colmajor_bf16(int64_t nn, const double* K64, __nv_bfloat16* out, cudaStream_t s) {
  if (nn <= 0) return cudaSuccess;
  if (nn * kNodeStrideC >= (int64_t(1) << 31)) return cudaErrorInvalidValue;
  stencil_colmajor_bf16_kernel<<<div_up(nn, kPackNodes), 256, 0, s>>>((int)nn, K64, out);
  return sf_launched(1);
}

__device__ __forceinline__ float bf16_lo(unsigned w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(unsigned w) { return __uint_as_float(w & 0xffff0000u); }

template <int EPI>
__global__ void __launch_bounds__(256) stencil_col_bf16_kernel(Grid g, FastDiv dz, FastDiv dy,
                                                               const __nv_bfloat16* __restrict__ coefC,
                                                               const uint8_t* __restrict__ mask,
                                                               const float* __restrict__ u, EpiArgs ea) {
  __shared__ float part[8][9][9];  // [warp][column][3 nodes x 3 rows]
  if (guard_off(ea.guard)) return;
  const int nn = (int)g.nn;
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int group = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);  // three nodes
  if (group * 3 >= nn) return;  // whole warps leave together
  // the row of this lane's sums
  const int dof = 9 * group + lane;
  const bool row = lane < 9 && dof < 3 * nn;
  float ob = 0.f, oi = 0.f, od = 0.f, xv = 0.f;
  uint8_t fr = 0;
  if (row) {
    fr = mask[dof];
    if (EPI != EPI_APPLY) ob = ((const float*)ea.b)[dof];
    if (EPI == EPI_CHEB1 || EPI == EPI_CHEB || EPI == EPI_JAC) oi = ((const float*)ea.dinv)[dof];
    if (EPI == EPI_CHEB) od = ((const float*)ea.d)[dof];
    if (EPI == EPI_CHEB1 || EPI == EPI_CHEB || EPI == EPI_JAC) xv = u[dof];
  }
  const int t = lane / 9, col = lane - 9 * t, n = group * 3 + t;
  if (lane < 27 && n < nn) {
    const uint4* cp = reinterpret_cast<const uint4*>(coefC) + (int64_t)group * 108 + lane;
    const uint4 q0 = cp[0], q1 = cp[27], q2 = cp[54], q3 = cp[81];
    const int NZ1 = g.nz + 1, NY1 = g.ny + 1;
    const int jq = (int)dz.div(n), k = n - jq * NZ1, i = (int)dy.div(jq), j = jq - i * NY1;
    const int ox = col / 3, oy = col - 3 * ox;
    // a neighbour outside the grid has zero coefficients: clamp it to the node itself
    const int dx = (ox == 0) ? (i > 0 ? -NY1 * NZ1 : 0) : (ox == 2 ? (i < g.nx ? NY1 * NZ1 : 0) : 0);
    const int dyo = (oy == 0) ? (j > 0 ? -NZ1 : 0) : (oy == 2 ? (j < g.ny ? NZ1 : 0) : 0);
    const int base = n + dx + dyo;
    const unsigned wv[16] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w,
                             q2.x, q2.y, q2.z, q2.w, q3.x, q3.y, q3.z, q3.w};
    float cf[28];
#pragma unroll
    for (int e = 0; e < 14; ++e) {
      cf[2 * e] = bf16_lo(wv[e]);
      cf[2 * e + 1] = bf16_hi(wv[e]);
    }
    float p0 = 0.f, p1 = 0.f, p2 = 0.f;
#pragma unroll
    for (int oz = 0; oz < 3; ++oz) {
      const int dzo = (oz == 0) ? (k > 0 ? -1 : 0) : (oz == 2 ? (k < g.nz ? 1 : 0) : 0);
      const float* um = u + 3 * (base + dzo);
      const float u0 = um[0], u1 = um[1], u2 = um[2];
      const float* c = cf + oz * 9;
      p0 = fmaf(c[0], u0, fmaf(c[1], u1, fmaf(c[2], u2, p0)));
      p1 = fmaf(c[3], u0, fmaf(c[4], u1, fmaf(c[5], u2, p1)));
      p2 = fmaf(c[6], u0, fmaf(c[7], u1, fmaf(c[8], u2, p2)));
    }
    part[wib][col][3 * t] = p0;
    part[wib][col][3 * t + 1] = p1;
    part[wib][col][3 * t + 2] = p2;
  }
  __syncwarp();
  if (!row) return;
  float ku = 0.f;
#pragma unroll
  for (int cc = 0; cc < 9; ++cc) ku += part[wib][cc][lane];
  const bool f = fr != 0;
  float* py = (EPI == EPI_APPLY || EPI == EPI_RESID ? (float*)ea.y : (float*)ea.xo) + dof;
  float res = 0.f, dn = 0.f;
  if (EPI == EPI_APPLY) {
    res = ku;
  } else if (EPI == EPI_RESID) {
    res = sub_rn(ob, ku);
  } else if (EPI == EPI_CHEB1) {
    dn = mul_rn(oi, sub_rn(ob, ku));
    res = add_rn(xv, mul_rn((float)ea.s1, dn));
  } else if (EPI == EPI_CHEB) {
    dn = mul_rn((float)ea.s1, add_rn(mul_rn(oi, sub_rn(ob, ku)), mul_rn((float)ea.s2, od)));
    res = add_rn(xv, dn);
  } else {
    res = add_rn(xv, mul_rn(mul_rn((float)ea.s1, oi), sub_rn(ob, ku)));
  }
  *py = f ? res : 0.f;
  if (EPI == EPI_CHEB1 || EPI == EPI_CHEB) ((float*)ea.d)[dof] = f ? dn : 0.f;
}

cudaError_t launch_stencil_col_bf16(Epi epi, const Grid& g, const __nv_bfloat16* coefC, const uint8_t* mask,
                                    const float* u, const EpiArgs& ea, cudaStream_t s) {
  if (3 * g.nn >= (int64_t(1) << 31) || g.nn * kNodeStrideC >= (int64_t(1) << 31)) return cudaErrorInvalidValue;
  const int nb = div_up(div_up(g.nn, 3), 8);
  const FastDiv dz = FastDiv::make(g.nz + 1), dy = FastDiv::make(g.ny + 1);
  switch (epi) {
    case EPI_APPLY: stencil_col_bf16_kernel<EPI_APPLY><<<nb, 256, 0, s>>>(g, dz, dy, coefC, mask, u, ea); break;
    case EPI_RESID: stencil_col_bf16_kernel<EPI_RESID><<<nb, 256, 0, s>>>(g, dz, dy, coefC, mask, u, ea); break;
    case EPI_CHEB1: stencil_col_bf16_kernel<EPI_CHEB1><<<nb, 256, 0, s>>>(g, dz, dy, coefC, mask, u, ea); break;
    case EPI_CHEB: stencil_col_bf16_kernel<EPI_CHEB><<<nb, 256, 0, s>>>(g, dz, dy, coefC, mask, u, ea); break;
    case EPI_JAC: stencil_col_bf16_kernel<EPI_JAC><<<nb, 256, 0, s>>>(g, dz, dy, coefC, mask, u, ea); break;
    default: return cudaErrorInvalidValue;
  }
  return sf_launched(1);
}

// ----------------------------------------------------------------------------
// Level-1 Galerkin operator from the fine element moduli: for every coarse
// element C and sub-element stu, E_fine[child(C, stu)] * Q_stu with
// Q_stu = P24(stu)^T KE P24(stu), child clamped to the fine grid exactly as
// gpu_fem/multigrid_v4.py:285-289 does.  Q is given in corner-major order
// Q[stu][(a * 3 + r) * 24 + b * 3 + q] with a, b coarse-element corners.
//
// A block makes one offset o of 128 coarse nodes.  A thread per (node, offset) with nine
// loads of Q from L1 for nine products and 64-bit divisions for the node's position took
// 151 us at 69,741 nodes (their 321 M FP64 products take 17); with the block's part of Q
// in shared memory and an element's eight moduli in flight together 100 (two nodes a
// thread, sharing the loads of Q: 108, for the registers).
constexpr int kL1Threads = 128;

__global__ void __launch_bounds__(kL1Threads) level1_assemble_kernel(Grid gc, Grid gf, FastDiv dz, FastDiv dy,
                                                                     const double* __restrict__ E,
                                                                     const double* __restrict__ Q,
                                                                     const uint8_t* __restrict__ mask,
                                                                     double* __restrict__ coef) {
  __shared__ __align__(16) double q[8 * 8 * 10];  // [a][stu][3 x 3, padded], corners a with node + o in the element
  const int o = blockIdx.y, ox = o / 9 - 1, oy = (o / 3) % 3 - 1, oz = o % 3 - 1;
  for (int e = threadIdx.x; e < 8 * 8 * 10; e += kL1Threads) {
    const int a = e / 80, stu = e / 10 % 8, r = e % 10;
    const int bx = (a >> 2) + ox, by = ((a >> 1) & 1) + oy, bz = (a & 1) + oz;
    const bool in = r < 9 && bx >= 0 && bx <= 1 && by >= 0 && by <= 1 && bz >= 0 && bz <= 1;
    q[(a * 8 + stu) * 10 + r] =
        in ? Q[(int64_t)stu * 576 + (a * 3 + r / 3) * 24 + (bx * 4 + by * 2 + bz) * 3 + r % 3] : 0.0;
  }
  __syncthreads();
  const int64_t n = (int64_t)blockIdx.x * kL1Threads + threadIdx.x;
  if (n >= gc.nn) return;
  int i, j, k;
  node_ijk(gc, dz, dy, (int)n, i, j, k);
  const int mi = i + ox, mj = j + oy, mk = k + oz;
  const bool ok = mi >= 0 && mj >= 0 && mk >= 0 && mi <= gc.nx && mj <= gc.ny && mk <= gc.nz;
  double blk[9];
#pragma unroll
  for (int r = 0; r < 9; ++r) blk[r] = 0.0;
  for (int a = 0; a < 8 && ok; ++a) {
    const int ax = a >> 2, ay = (a >> 1) & 1, az = a & 1;
    const int bx = ax + ox, by = ay + oy, bz = az + oz;
    if (bx < 0 || bx > 1 || by < 0 || by > 1 || bz < 0 || bz > 1) continue;
    const int ci = i - ax, cj = j - ay, ck = k - az;
    // no branch around the loads: one corner's fly while the last one's products run
    const bool in = ci >= 0 && cj >= 0 && ck >= 0 && ci < gc.nx && cj < gc.ny && ck < gc.nz;
    double Ee[8], elem[9];
#pragma unroll
    for (int stu = 0; stu < 8; ++stu) {
      const int fi = min(2 * ci + (stu >> 2), gf.nx - 1);
      const int fj = min(2 * cj + ((stu >> 1) & 1), gf.ny - 1);
      const int fk = min(2 * ck + (stu & 1), gf.nz - 1);
      Ee[stu] = in ? E[((int64_t)fi * gf.ny + fj) * gf.nz + fk] : 0.0;
    }
#pragma unroll
    for (int r = 0; r < 9; ++r) elem[r] = 0.0;
#pragma unroll
    for (int stu = 0; stu < 8; ++stu) {
      double qv[10];
#pragma unroll
      for (int r = 0; r < 10; r += 2) {
        const double2 v = *reinterpret_cast<const double2*>(q + (a * 8 + stu) * 10 + r);
        qv[r] = v.x;
        qv[r + 1] = v.y;
      }
#pragma unroll
      for (int r = 0; r < 9; ++r) elem[r] = fma(Ee[stu], qv[r], elem[r]);
    }
    if (in) {
#pragma unroll
      for (int r = 0; r < 9; ++r) blk[r] += elem[r];
    }
  }
  const int64_t m = ok ? node_id(gc, mi, mj, mk) : 0;
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const bool keep = ok && mask[3 * n + r] && mask[3 * m + c];
      coef[((int64_t)o * 9 + r * 3 + c) * gc.nn + n] = keep ? blk[r * 3 + c] : 0.0;
    }
}

cudaError_t launch_level1_assemble(const Grid& gc, const Grid& gf, const double* E_fine,
                                   const double* Q, const uint8_t* mask_c, double* coef,
                                   cudaStream_t s) {
  if (gc.nn >= (int64_t(1) << 31)) return cudaErrorInvalidValue;
  const FastDiv dz = FastDiv::make(gc.nz + 1), dy = FastDiv::make(gc.ny + 1);
  level1_assemble_kernel<<<dim3(div_up(gc.nn, kL1Threads), 27), kL1Threads, 0, s>>>(gc, gf, dz, dy, E_fine, Q, mask_c,
                                                                                    coef);
  return sf_launched(1);
}

// ----------------------------------------------------------------------------
// 1-D trilinear weights, row-normalised as in gpu_fem/solver_v2.py:62-149:
// w[3 * f + (f - 2 * c + 1)] is the weight of coarse node c for fine node f.
__device__ __forceinline__ double w1(const double* w, int f, int c) {
  const int d = f - 2 * c;
  return (d < -1 || d > 1) ? 0.0 : w[3 * f + d + 1];
}

// K_c = R K_f P on stencils (Galerkin triple product of the reference's RAP loop).
// Coarse block (n, M = n + o) = sum over fine nodes f in the support of n and
// fine neighbours g = f + d of f in the support of M of
// P[f, n] K_f[f, g] P[g, M].  The trilinear weights factor per axis: with f = 2 I + a - 1
// and g = f + d - 1 (a, d = 0..2), g supports I + m where a + d is 0 or 1 for m = -1, 1
// to 3 for m = 0 and 3 or 4 for m = 1, and the sum runs over the product of the axes'
// pairs, x outermost, in ascending (a, d).
//
// One thread per coarse node, entry r of the 3 x 3 block and (mx, my), all three mz: a
// warp is 32 nodes along z, the nine warps of a block the nine (mx, my) of one entry,
// whose fine coefficients (126 KB) its L1 holds.  An x pair's y pairs are straight-line
// code (MY), nine loads each that the three mz share.  A thread per block with all
// nine entries chained up to 343 x 9 loads: 140 us each for the 1,386 and the 168
// coarse nodes of 80 x 40 x 20 (two levels), 241 for the two of 160 x 80 x 40, 341 of
// 200 x 100 x 50; now 23, 98 and 179.  Two blocks per SM at 96 registers spill 56 bytes
// and are faster than one at 134 (122 and 228).
__host__ __device__ constexpr bool rap_pair(int a, int d, int m) {
  return m < 0 ? a + d <= 1 : (m > 0 ? a + d >= 3 : a + d >= 1 && a + d <= 3);
}
// w(f, I) w(g, I + m) of pair (a, d); zero where a node is missing
__device__ __forceinline__ double rap_weight(const double* __restrict__ w, int I, int m, int nf, int nc, int a, int d) {
  const int f = 2 * I + a - 1, gg = f + d - 1, c = I + m;
  if (f < 0 || f > nf || gg < 0 || gg > nf || c < 0 || c > nc) return 0.0;
  return w[3 * f + a] * w1(w, gg, c);
}

// base: entry r of the fine node (2I, 2J, 2K), stencil block of offset (0, 0, 0);
// block (dx, dy, dz) lies (dx * 9 + dy * 3 + dz) * 9 * nn further
template <int MY>
__device__ __forceinline__ void rap_sum(const Grid& gf, const Grid& gc, const double* __restrict__ base,
                                        const double* __restrict__ wx, const double* __restrict__ wy,
                                        const double* __restrict__ wz, int I, int J, int K, int mx, double (&acc)[3]) {
  const int64_t nn = gf.nn, ys = gf.nz + 1, xs = (gf.ny + 1) * ys;
  double pz[3][3][3], py[3][3];  // [m + 1][a][d], [a][d]; entries outside rap_pair are not used
  bool fz[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    fz[a] = 2 * K + a - 1 >= 0 && 2 * K + a - 1 <= gf.nz;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      if (rap_pair(a, d, MY)) py[a][d] = rap_weight(wy, J, MY, gf.ny, gc.ny, a, d);
#pragma unroll
      for (int m = 0; m < 3; ++m)
        if (rap_pair(a, d, m - 1)) pz[m][a][d] = rap_weight(wz, K, m - 1, gf.nz, gc.nz, a, d);
    }
  }
  for (int ex = 0; ex < 9; ++ex) {
    const int ax = ex / 3, dx = ex % 3;
    if (!rap_pair(ax, dx, mx)) continue;
    const double px = rap_weight(wx, I, mx, gf.nx, gc.nx, ax, dx);
    if (px == 0.0) continue;
    const double* bx = base + (ax - 1) * xs + dx * 81 * nn;
#pragma unroll
    for (int ay = 0; ay < 3; ++ay)
#pragma unroll
      for (int dy = 0; dy < 3; ++dy)
        if (rap_pair(ay, dy, MY)) {
          const double pxy = px * py[ay][dy];
          const double* bxy = bx + (ay - 1) * ys + dy * 27 * nn;
          double v[3][3];
#pragma unroll
          for (int d = 0; d < 3; ++d)
#pragma unroll
            for (int a = 0; a < 3; ++a) v[a][d] = fz[a] && pxy != 0.0 ? bxy[d * 9 * nn + a - 1] : 0.0;
#pragma unroll
          for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int d = 0; d < 3; ++d) {
              const double pv = pxy * v[a][d];  // exact: the weights are powers of two
#pragma unroll
              for (int m = 0; m < 3; ++m)
                if (rap_pair(a, d, m - 1)) acc[m] = fma(pz[m][a][d], pv, acc[m]);
            }
        }
  }
}

__global__ void __launch_bounds__(288, 2) rap_kernel(Grid gf, Grid gc, FastDiv dz, FastDiv dy,
                                                     const double* __restrict__ cf,
                                                     const uint8_t* __restrict__ mask_c,
                                                     const double* __restrict__ wx, const double* __restrict__ wy,
                                                     const double* __restrict__ wz, double* __restrict__ cc) {
  const int64_t n = (int64_t)blockIdx.x * 32 + (threadIdx.x & 31);
  if (n >= gc.nn) return;
  const int r = blockIdx.y, warp = threadIdx.x >> 5, mx = warp / 3 - 1, my = warp % 3 - 1;
  int I, J, K;
  node_ijk(gc, dz, dy, (int)n, I, J, K);
  const bool col = I + mx >= 0 && I + mx <= gc.nx && J + my >= 0 && J + my <= gc.ny;
  double acc[3] = {0.0, 0.0, 0.0};
  if (col) {
    const double* base = cf + r * gf.nn + node_id(gf, 2 * I, 2 * J, 2 * K);
    if (my < 0) rap_sum<-1>(gf, gc, base, wx, wy, wz, I, J, K, mx, acc);
    else if (my > 0) rap_sum<1>(gf, gc, base, wx, wy, wz, I, J, K, mx, acc);
    else rap_sum<0>(gf, gc, base, wx, wy, wz, I, J, K, mx, acc);
  }
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    const int MK = K + m - 1;
    bool keep = col && MK >= 0 && MK <= gc.nz;
    if (keep) keep = mask_c[3 * n + r / 3] && mask_c[3 * node_id(gc, I + mx, J + my, MK) + r % 3];
    cc[((int64_t)((mx + 1) * 9 + (my + 1) * 3 + m) * 9 + r) * gc.nn + n] = keep ? acc[m] : 0.0;
  }
}

cudaError_t launch_rap(const Grid& gf, const Grid& gc, const double* coef_f, const uint8_t* mask_c,
                       const double* wx, const double* wy, const double* wz, double* coef_c,
                       cudaStream_t s) {
  if (gc.nn >= (int64_t(1) << 31)) return cudaErrorInvalidValue;
  const FastDiv dz = FastDiv::make(gc.nz + 1), dy = FastDiv::make(gc.ny + 1);
  rap_kernel<<<dim3(div_up(gc.nn, 32), 9), 288, 0, s>>>(gf, gc, dz, dy, coef_f, mask_c, wx, wy, wz, coef_c);
  return sf_launched(1);
}

__global__ void stencil_diag_kernel(Grid g, const double* __restrict__ coef, const uint8_t* __restrict__ mask,
                                    double* __restrict__ dinv) {
  const int64_t dof = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (dof >= g.ndof) return;
  const int64_t n = dof / 3;
  const int r = (int)(dof - 3 * n);
  double d = coef[((int64_t)13 * 9 + r * 3 + r) * g.nn + n];
  d = fabs(d) > 1e-12 ? d : 1.0;
  dinv[dof] = mask[dof] ? 1.0 / d : 0.0;
}

cudaError_t launch_stencil_diag(const Grid& g, const double* coef, const uint8_t* mask,
                                double* dinv, cudaStream_t s) {
  stencil_diag_kernel<<<div_up(g.ndof, 256), 256, 0, s>>>(g, coef, mask, dinv);
  return sf_launched(1);
}

// ----------------------------------------------------------------------------
// Weights of fine nodes 2 I - 1 .. 2 I + 1 for coarse node I along one axis (0 outside
// the grid).  Row-normalised trilinear weights are 0, 1/2 or 1, so their products are
// exact in either type.
template <typename T>
__device__ __forceinline__ void axis_weights(const double* __restrict__ w, int I, int nf, T (&out)[3]) {
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int f = 2 * I + a - 1;
    out[a] = (f < 0 || f > nf) ? T(0) : (T)w[3 * f + a];
  }
}

// One thread per coarse DOF (a thread per node kept 74 blocks of 128 busy on the
// 9,471-node level of 80 x 40 x 20: 8.8 us).  With a zero start requested the level's
// first smoothing step, which only scales the restricted residual, is formed here.
template <typename T>
__global__ void __launch_bounds__(256) restrict_kernel(Grid gf, Grid gc, FastDiv dz, FastDiv dy,
                                                       const double* __restrict__ wx, const double* __restrict__ wy,
                                                       const double* __restrict__ wz,
                                                       const uint8_t* __restrict__ mask_c, const T* __restrict__ fine,
                                                       T* __restrict__ coarse, ZeroStart zs, const int* guard) {
  if (guard_off(guard)) return;
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= 3 * gc.nn) return;
  const int n = (int)(idx / 3), c = (int)(idx - 3 * (int64_t)n);
  const int NZc = gc.nz + 1, NYc = gc.ny + 1, NZ = gf.nz + 1, NY = gf.ny + 1;
  const int jq = (int)dz.div(n), K = n - jq * NZc, I = (int)dy.div(jq), J = jq - I * NYc;
  T px[3], py[3], pz[3];
  axis_weights(wx, I, gf.nx, px);
  axis_weights(wy, J, gf.ny, py);
  axis_weights(wz, K, gf.nz, pz);
  const T* f0 = fine + 3 * (((int64_t)(2 * I) * NY + 2 * J) * NZ + 2 * K) + c;
  T v[27];
#pragma unroll
  for (int d = 0; d < 27; ++d) {
    const int ax = d / 9, ay = (d / 3) % 3, az = d % 3;
    const T p = px[ax] * py[ay] * pz[az];
    v[d] = p != T(0) ? f0[3 * (((int64_t)(ax - 1) * NY + (ay - 1)) * NZ + az - 1)] : T(0);
  }
  T acc = T(0);
#pragma unroll
  for (int d = 0; d < 27; ++d) {
    const T p = px[d / 9] * py[(d / 3) % 3] * pz[d % 3];
    if (p != T(0)) acc += p * v[d];
  }
  const T r = mask_c[idx] ? acc : T(0);
  coarse[idx] = r;
  zero_start<T>(zs, idx, r);
}

// One thread per fine node; ADD: x += P e (with e's prolongation rounded first, as a
// separate correction vector would be), else x = P e.  (A thread per DOF spends three
// times the index and weight instructions, which bind it: 15.5 us a level of
// 200 x 100 x 50 on average against 7.9 and 6.1 for P e and the sum by themselves.)
template <typename T, bool ADD>
__global__ void __launch_bounds__(256) prolong_kernel(Grid gf, Grid gc, FastDiv dz, FastDiv dy,
                                                      const double* __restrict__ wx, const double* __restrict__ wy,
                                                      const double* __restrict__ wz,
                                                      const uint8_t* __restrict__ mask_f, const T* __restrict__ coarse,
                                                      T* __restrict__ fine, const int* guard) {
  if (guard_off(guard)) return;
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= gf.nn) return;
  const int f = (int)idx;
  const int NZc = gc.nz + 1, NYc = gc.ny + 1, NZ = gf.nz + 1, NY = gf.ny + 1;
  const int jq = (int)dz.div(f), k = f - jq * NZ, i = (int)dy.div(jq), j = jq - i * NY;
  T x[3];
  bool fr[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    x[c] = ADD ? fine[3 * (int64_t)f + c] : T(0);
    fr[c] = mask_f[3 * (int64_t)f + c] != 0;
  }
  // coarse parents floor(i/2) and floor(i/2) + 1 per axis, weights 0 where there is none
  T qx[2], qy[2], qz[2];
#pragma unroll
  for (int b = 0; b < 2; ++b) {
    const int I = (i >> 1) + b, J = (j >> 1) + b, K = (k >> 1) + b;
    qx[b] = I > gc.nx ? T(0) : (T)w1(wx, i, I);
    qy[b] = J > gc.ny ? T(0) : (T)w1(wy, j, J);
    qz[b] = K > gc.nz ? T(0) : (T)w1(wz, k, K);
  }
  const T* c0 = coarse + 3 * (((int64_t)(i >> 1) * NYc + (j >> 1)) * NZc + (k >> 1));
  T v[8][3];
#pragma unroll
  for (int a = 0; a < 8; ++a) {
    const T p = qx[a >> 2] * qy[(a >> 1) & 1] * qz[a & 1];
    const T* ca = c0 + 3 * ((a >> 2) * NYc * NZc + ((a >> 1) & 1) * NZc + (a & 1));
#pragma unroll
    for (int c = 0; c < 3; ++c) v[a][c] = p != T(0) ? ca[c] : T(0);
  }
  T acc[3] = {T(0), T(0), T(0)};
#pragma unroll
  for (int a = 0; a < 8; ++a) {
    const T p = qx[a >> 2] * qy[(a >> 1) & 1] * qz[a & 1];
    if (p != T(0)) {
#pragma unroll
      for (int c = 0; c < 3; ++c) acc[c] += p * v[a][c];
    }
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const T e = fr[c] ? acc[c] : T(0);
    fine[3 * (int64_t)f + c] = ADD ? add_rn(x[c], e) : e;
  }
}

cudaError_t launch_restrict(DType t, const Grid& gf, const Grid& gc, const double* wx,
                            const double* wy, const double* wz, const uint8_t* mask_c,
                            const void* fine, void* coarse, const int* guard, cudaStream_t s, const ZeroStart& zs) {
  if (gc.nn >= (int64_t(1) << 31)) return cudaErrorInvalidValue;
  const int nb = div_up(3 * gc.nn, 256);
  const FastDiv dz = FastDiv::make(gc.nz + 1), dy = FastDiv::make(gc.ny + 1);
  if (t == F64)
    restrict_kernel<double><<<nb, 256, 0, s>>>(gf, gc, dz, dy, wx, wy, wz, mask_c, (const double*)fine,
                                               (double*)coarse, zs, guard);
  else
    restrict_kernel<float><<<nb, 256, 0, s>>>(gf, gc, dz, dy, wx, wy, wz, mask_c, (const float*)fine,
                                              (float*)coarse, zs, guard);
  return sf_launched(1);
}

cudaError_t launch_prolong(DType t, const Grid& gf, const Grid& gc, const double* wx,
                           const double* wy, const double* wz, const uint8_t* mask_f,
                           const void* coarse, void* fine, bool add, const int* guard, cudaStream_t s) {
  if (gf.nn >= (int64_t(1) << 31)) return cudaErrorInvalidValue;
  const int nb = div_up(gf.nn, 256);
  const FastDiv dz = FastDiv::make(gf.nz + 1), dy = FastDiv::make(gf.ny + 1);
#define SF_PROLONG(T, A) \
  prolong_kernel<T, A><<<nb, 256, 0, s>>>(gf, gc, dz, dy, wx, wy, wz, mask_f, (const T*)coarse, (T*)fine, guard)
  if (t == F64) {
    if (add) SF_PROLONG(double, true);
    else SF_PROLONG(double, false);
  } else {
    if (add) SF_PROLONG(float, true);
    else SF_PROLONG(float, false);
  }
#undef SF_PROLONG
  return sf_launched(1);
}

// ----------------------------------------------------------------------------
// Dense free-DOF matrix of the coarsest stencil (row-major n x n; A zeroed first).
__global__ void stencil_to_dense_kernel(Grid g, const double* __restrict__ coef,
                                        const int32_t* __restrict__ didx, int64_t n,
                                        double* __restrict__ A) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= 27 * g.ndof) return;
  const int o = (int)(idx / g.ndof);
  const int64_t dof = idx - (int64_t)o * g.ndof;
  const int64_t p = didx[dof];
  if (p < 0) return;
  const int64_t node = dof / 3;
  const int r = (int)(dof - 3 * node);
  int i, j, k;
  node_ijk(g, node, i, j, k);
  const int mi = i + o / 9 - 1, mj = j + (o / 3) % 3 - 1, mk = k + o % 3 - 1;
  if (mi < 0 || mj < 0 || mk < 0 || mi > g.nx || mj > g.ny || mk > g.nz) return;
  const int64_t m = node_id(g, mi, mj, mk);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const int64_t q = didx[3 * m + c];
    if (q < 0) continue;
    A[p * n + q] = coef[((int64_t)o * 9 + r * 3 + c) * g.nn + node];
  }
}

cudaError_t launch_stencil_to_dense(const Grid& g, const double* coef, const int32_t* dense_idx,
                                    int64_t n, double* A, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(A, 0, sizeof(double) * n * n, s);
  if (e != cudaSuccess) return e;
  stencil_to_dense_kernel<<<div_up(27 * g.ndof, 256), 256, 0, s>>>(g, coef, dense_idx, n, A);
  return sf_launched(1);
}

// ----------------------------------------------------------------------------
template <typename A, typename B>
__global__ void convert_kernel(const A* __restrict__ src, B* __restrict__ dst, int64_t n, const int* guard) {
  if (guard_off(guard)) return;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = from_d<B>(to_d(src[i]));
}

template <>
__global__ void convert_kernel<double, float>(const double* __restrict__ src, float* __restrict__ dst,
                                              int64_t n, const int* guard) {
  if (guard_off(guard)) return;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = __double2float_rn(src[i]);
}

__global__ void __launch_bounds__(256) convert_start_kernel(int64_t n, const double* __restrict__ src,
                                                            float* __restrict__ dst, ZeroStart zs, const int* guard) {
  if (guard_off(guard)) return;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float v = __double2float_rn(src[i]);
  dst[i] = v;
  zero_start<float>(zs, i, v);
}

cudaError_t launch_convert_start(int64_t n, const double* src, float* dst, const ZeroStart& zs, const int* guard,
                                 cudaStream_t s) {
  convert_start_kernel<<<div_up(n, 256), 256, 0, s>>>(n, src, dst, zs, guard);
  return sf_launched(1);
}

cudaError_t launch_convert(DType from, DType to, const void* src, void* dst, int64_t n,
                           const int* guard, cudaStream_t s) {
  const int nb = div_up(n, 256);
  if (from == F64 && to == F32)
    convert_kernel<double, float><<<nb, 256, 0, s>>>((const double*)src, (float*)dst, n, guard);
  else if (from == F32 && to == F64)
    convert_kernel<float, double><<<nb, 256, 0, s>>>((const float*)src, (double*)dst, n, guard);
  else if (from == F64 && to == BF16)
    convert_kernel<double, __nv_bfloat16><<<nb, 256, 0, s>>>((const double*)src,
                                                             (__nv_bfloat16*)dst, n, guard);
  else if (from == F64 && to == F64)
    convert_kernel<double, double><<<nb, 256, 0, s>>>((const double*)src, (double*)dst, n, guard);
  else if (from == F32 && to == F32)
    convert_kernel<float, float><<<nb, 256, 0, s>>>((const float*)src, (float*)dst, n, guard);
  else
    return cudaErrorInvalidValue;
  return sf_launched(1);
}

}  // namespace simpfem
