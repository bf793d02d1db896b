// Fine-level hex8 operator for the structured SIMP mesh.
//
// Replaces the reference's MatrixFreeKff.matvec (gpu_fem/solver_v2.py:1182-1222:
// expand -> gather -> KE @ u_elem.T * E -> bincount -> restrict) and the fused
// FusedMatvec kernels (gpu_fem/cuda_fused_matvec.py:41-88, :112-246) with one
// deterministic sweep kernel:
//
//  * Node indices are computed from (i, j, k); there is no edof table.
//  * A block owns a (bj-1) x (bk-1) patch of node columns (one halo element
//    column on the low j and k sides) and sweeps cx node planes along x, so
//    every element is evaluated once per sweep (plus the halo columns).
//  * The element product KE * u_e uses the reflection symmetry of the unit
//    cube: in the Walsh (+/-1) basis over the element's 2x2x2 nodes the 24x24
//    unit stiffness is block diagonal with eight 3x3 blocks, of which six couple
//    only two of their three modes (an isotropic material; checked when the
//    stiffness is installed): 48 products instead of 576.  The transform is
//    separable, so a node plane is transformed along y and z once for the two
//    element planes it bounds, and the two face sums that meet on it are added
//    before they are transformed back.
//  * Per-node sums are reduced in shared memory in a fixed order (no atomics),
//    and the caller's epilogue (residual, Chebyshev or Jacobi update) is fused
//    into the store.
#include <stdio.h>

#include "common.cuh"
#include "gmg_impl.h"

namespace simpfem {

__constant__ double c_wht64[8][9];
__constant__ float2 c_wht32[4][9];   // FP32 blocks 2h and 2h + 1 as the lanes of a pair
__constant__ float2 c_whtb32[4][9];  // the same for KE with its entries rounded to bf16
__constant__ double c_kediag[24];  // KE diagonal, corner-major order
__constant__ double c_kenb[8][9];  // 3x3 node-diagonal blocks of KE per corner

// corner q = dx * 4 + dy * 2 + dz  <->  reference local node (gpu_fem/pub_simp_solver.py:196-207)
static const int kRefNodeOfCorner[8] = {0, 4, 3, 7, 1, 5, 2, 6};

// Pattern of the Walsh blocks of an isotropic stiffness: blocks 0 and 7 are full,
// the others couple two modes and leave the third (lone_mode) by itself.
__host__ __device__ constexpr int lone_mode(int b) { return b == 1 || b == 6 ? 2 : (b == 2 || b == 5 ? 1 : 0); }
__host__ __device__ constexpr bool block_entry(int b, int r, int c) {
  return b == 0 || b == 7 || r == c || (r != lone_mode(b) && c != lone_mode(b));
}
static bool has_pattern(const WhtBlocks& wb) {
  double mx = 0.0, off = 0.0;
  for (int b = 0; b < 8; ++b)
    for (int i = 0; i < 9; ++i) {
      const double v = fabs(wb.b[b][i]);
      mx = v > mx ? v : mx;
      if (!block_entry(b, i / 3, i % 3)) off = v > off ? v : off;
    }
  return off <= 1e-15 * mx;  // a few roundings of the largest entry
}
// Whether the stiffness installed on a device has the pattern (FP64 products skip the
// other entries; the packed FP32 ones pair two blocks and take them all); written
// with the constants, which all meshes of a device share.
static std::atomic<int> g_pattern[64];
static bool pattern_on_device() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  return dev < 64 && g_pattern[dev].load(std::memory_order_acquire) != 0;
}

void set_fine_constants(const double* ke576, const WhtBlocks& wb) {
  // KE in corner-major order: row (q * 3 + c) <- reference row (3 * a(q) + c)
  double kem[576];
  for (int q = 0; q < 8; ++q)
    for (int c = 0; c < 3; ++c)
      for (int q2 = 0; q2 < 8; ++q2)
        for (int c2 = 0; c2 < 3; ++c2)
          kem[(q * 3 + c) * 24 + q2 * 3 + c2] =
              ke576[(3 * kRefNodeOfCorner[q] + c) * 24 + 3 * kRefNodeOfCorner[q2] + c2];
  // KE with bf16-rounded entries has Walsh blocks of its own as long as mirrored entries
  // round alike.  An accepted KE may be off its reflection symmetry by up to 1e-9, and
  // entries on two sides of a rounding boundary would then part by 2^-8, terms that the
  // blocks cannot hold: so the entries of corner 0 are rounded and mirrored.
  double keb[576];
  for (int q = 0; q < 8; ++q)
    for (int c = 0; c < 3; ++c)
      for (int q2 = 0; q2 < 8; ++q2)
        for (int c2 = 0; c2 < 3; ++c2) {
          const bool odd = ((q & (4 >> c)) != 0) != ((q & (4 >> c2)) != 0);  // a component changes sign along its own axis
          const double v = ke576[(3 * kRefNodeOfCorner[0] + c) * 24 + 3 * kRefNodeOfCorner[q ^ q2] + c2];
          const double r = (double)__bfloat162float(__float2bfloat16_rn((float)v));
          keb[(3 * kRefNodeOfCorner[q] + c) * 24 + 3 * kRefNodeOfCorner[q2] + c2] = odd ? -r : r;
        }
  double boff = 0.0;
  const WhtBlocks wbb = make_wht_blocks(keb, &boff);
  double kd[24];
  for (int i = 0; i < 24; ++i) kd[i] = kem[i * 24 + i];
  double nb[8][9];
  for (int q = 0; q < 8; ++q)
    for (int r = 0; r < 3; ++r)
      for (int c = 0; c < 3; ++c) nb[q][r * 3 + c] = kem[(q * 3 + r) * 24 + q * 3 + c];
  float2 w32[4][9], wb32[4][9];
  for (int h = 0; h < 4; ++h)
    for (int i = 0; i < 9; ++i) {
      w32[h][i] = make_float2((float)wb.b[2 * h][i], (float)wb.b[2 * h + 1][i]);
      wb32[h][i] = make_float2((float)wbb.b[2 * h][i], (float)wbb.b[2 * h + 1][i]);
    }
  SF_CUDA(cudaMemcpyToSymbol(c_wht64, wb.b, sizeof(wb.b)));
  SF_CUDA(cudaMemcpyToSymbol(c_wht32, w32, sizeof(w32)));
  SF_CUDA(cudaMemcpyToSymbol(c_whtb32, wb32, sizeof(wb32)));
  SF_CUDA(cudaMemcpyToSymbol(c_kediag, kd, sizeof(kd)));
  SF_CUDA(cudaMemcpyToSymbol(c_kenb, nb, sizeof(nb)));
  int dev = 0;
  SF_CUDA(cudaGetDevice(&dev));
  if (dev < 64) g_pattern[dev].store(has_pattern(wb) ? 1 : 0, std::memory_order_release);
}

__device__ __forceinline__ void wht8(double a[8]) {
#pragma unroll
  for (int m = 4; m >= 1; m >>= 1) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      if ((q & m) == 0) {
        const double p = a[q], r = a[q | m];
        a[q] = p + r;
        a[q | m] = p - r;
      }
    }
  }
}

// f = KE * u for one element, u/f indexed [corner][component].
__device__ __forceinline__ void elem_wht(const double (&u)[8][3], double (&f)[8][3]) {
  double w[3][8];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
#pragma unroll
    for (int q = 0; q < 8; ++q) w[c][q] = u[q][c];
    wht8(w[c]);
  }
  double v[3][8];
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    const double in0 = w[0][b ^ 4], in1 = w[1][b ^ 2], in2 = w[2][b ^ 1];
    v[0][b ^ 4] = c_wht64[b][0] * in0 + c_wht64[b][1] * in1 + c_wht64[b][2] * in2;
    v[1][b ^ 2] = c_wht64[b][3] * in0 + c_wht64[b][4] * in1 + c_wht64[b][5] * in2;
    v[2][b ^ 1] = c_wht64[b][6] * in0 + c_wht64[b][7] * in1 + c_wht64[b][8] * in2;
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    wht8(v[c]);
#pragma unroll
    for (int q = 0; q < 8; ++q) f[q][c] = v[c][q];
  }
}

// FP32 runs on the packed pair instructions of sm_100 (half the issue slots), the
// lanes of a pair being z: the nodes dz = 0, 1 of a corner pair, or the z parities
// 0, 1 of a transformed value.  Only the z butterflies cross lanes.  Block b pairs
// value b ^ 4 of component 0 with b ^ 2 of component 1 and b ^ 1 of component 2, so
// with component 2 kept in swapped lanes blocks 2h and 2h + 1 are one pair.
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ float2 zbutterfly(float2 a) { return make_float2(__fadd_rn(a.x, a.y), __fsub_rn(a.x, a.y)); }
__device__ __forceinline__ float2 swap2(float2 a) { return make_float2(a.y, a.x); }

// The eight blocks: w[c][2 sx + sy] (component 2 swapped) -> v in the same layout.
// A row is a product and two fused multiply-adds; the element form begins with the
// second term, the face form with the first.
template <bool FACES, bool BF>
__device__ __forceinline__ void blocks2(const float2 (&w)[3][4], float2 (&v)[3][4]) {
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    const float2 in0 = w[0][h ^ 2], in1 = w[1][h ^ 1], in2 = w[2][h];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      const float2* c = BF ? c_whtb32[h] : c_wht32[h];
      float2 a;
      if (FACES) {
        a = __fmul2_rn(c[3 * r], in0);
        a = __ffma2_rn(c[3 * r + 1], in1, a);
      } else {
        a = __fmul2_rn(c[3 * r + 1], in1);
        a = __ffma2_rn(c[3 * r], in0, a);
      }
      a = __ffma2_rn(c[3 * r + 2], in2, a);
      v[r][r == 0 ? h ^ 2 : (r == 1 ? h ^ 1 : h)] = a;
    }
  }
}

// f = E * KE * u for one element: lo and hi are its faces at dx = 0 and 1, node pairs
// [component][dy].  The modulus is contracted into the first back-transform butterfly.
__device__ __forceinline__ void element_product2(const float2 (&ulo)[3][2], const float2 (&uhi)[3][2], float E,
                                                 float2 (&flo)[3][2], float2 (&fhi)[3][2]) {
  float2 w[3][4], v[3][4];
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const float2 s0 = add2(ulo[q][0], uhi[q][0]), s1 = add2(ulo[q][1], uhi[q][1]);
    const float2 d0 = sub2(ulo[q][0], uhi[q][0]), d1 = sub2(ulo[q][1], uhi[q][1]);
    w[q][0] = zbutterfly(add2(s0, s1));
    w[q][1] = zbutterfly(sub2(s0, s1));
    w[q][2] = zbutterfly(add2(d0, d1));
    w[q][3] = zbutterfly(sub2(d0, d1));
    if (q == 2) {
#pragma unroll
      for (int s = 0; s < 4; ++s) w[q][s] = swap2(w[q][s]);
    }
  }
  blocks2<false, false>(w, v);
  const float2 E2 = make_float2(E, E);
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    float2 s[2], d[2];
#pragma unroll
    for (int y = 0; y < 2; ++y) {
      const float2 r = __fmul2_rn(E2, v[q][2 + y]);
      s[y] = __ffma2_rn(E2, v[q][y], r);
      d[y] = __ffma2_rn(E2, v[q][y], make_float2(-r.x, -r.y));
    }
    const float2 a0 = add2(s[0], s[1]), a1 = sub2(s[0], s[1]), b0 = add2(d[0], d[1]), b1 = sub2(d[0], d[1]);
    flo[q][0] = zbutterfly(q == 2 ? swap2(a0) : a0);
    flo[q][1] = zbutterfly(q == 2 ? swap2(a1) : a1);
    fhi[q][0] = zbutterfly(q == 2 ? swap2(b0) : b0);
    fhi[q][1] = zbutterfly(q == 2 ? swap2(b1) : b1);
  }
}

// The same in FP64; faces are node values [component][2 dy + dz].  All entries are
// taken: those outside the pattern can hold roundings of the transform.  They come
// from shared memory (cw: ten values a block): constants are hoisted out of the
// plane loop into registers, 144 of them (512k elements: 47 us at two blocks per SM,
// 37 so at three).
constexpr int kBlockCoefs = 10;
__device__ __forceinline__ void element_product(const double (&ulo)[3][4], const double (&uhi)[3][4], double E,
                                                const double* cw, double (&flo)[3][4], double (&fhi)[3][4]) {
  double w[3][8], v[3][8];
#pragma unroll
  for (int q = 0; q < 3; ++q) {
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      w[q][s] = ulo[q][s];
      w[q][4 + s] = uhi[q][s];
    }
    wht8(w[q]);
  }
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    const double in[3] = {w[0][b ^ 4], w[1][b ^ 2], w[2][b ^ 1]};
    double co[kBlockCoefs];
#pragma unroll
    for (int k = 0; k < kBlockCoefs; k += 2) {
      const double2 c = *reinterpret_cast<const double2*>(cw + b * kBlockCoefs + k);
      co[k] = c.x;
      co[k + 1] = c.y;
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      double acc = mul_rn(co[3 * r + 1], in[1]);
      acc = fma(co[3 * r], in[0], acc);
      acc = fma(co[3 * r + 2], in[2], acc);
      v[r][b ^ (4 >> r)] = acc;
    }
  }
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    double f[8];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const double r = mul_rn(E, v[q][4 + s]);
      f[s] = fma(E, v[q][s], r);
      f[4 + s] = fma(E, v[q][s], -r);
    }
#pragma unroll
    for (int m = 2; m >= 1; m >>= 1)
#pragma unroll
      for (int s = 0; s < 8; ++s)
        if ((s & m) == 0) {
          const double a = f[s], b = f[s | m];
          f[s] = a + b;
          f[s | m] = a - b;
        }
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      flo[q][s] = f[s];
      fhi[q][s] = f[4 + s];
    }
  }
}

// One value copied global -> shared asynchronously (cp.async; zero-filled when ok
// is false, reading nothing from src, which is then any valid address).
template <typename T>
__device__ __forceinline__ void cp_async_elem(T* dst, const T* src, bool ok) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  if (sizeof(T) == 8)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(ok ? 8 : 0));
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(d), "l"(src), "r"(ok ? 4 : 0));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
__device__ __forceinline__ void cp_async_wait_all_but_one() { asm volatile("cp.async.wait_group 1;\n" ::); }

// One face of an element column at a node plane (12 values): with FORM kFaces
// transformed along z and y -- v[component][2 a + b], a the y and b the z parity
// (FP32: component 2 with b swapped) --, else its node values v[component][2 dy + dz].
enum SweepForm { kFaces = 0, kElement = 1 };

template <bool BF, int FORM>
__device__ __forceinline__ void face_values(const double* r0, const double* r1, double (&v)[3][4], double (&own)[3]) {
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    own[q] = r0[q];
    const double n00 = own[q], n01 = r0[3 + q], n10 = r1[q], n11 = r1[3 + q];
    if (FORM != kFaces) {
      v[q][0] = n00;
      v[q][1] = n01;
      v[q][2] = n10;
      v[q][3] = n11;
      continue;
    }
    const double s0 = n00 + n01, d0 = n00 - n01, s1 = n10 + n11, d1 = n10 - n11;
    v[q][0] = s0 + s1;
    v[q][1] = d0 + d1;
    v[q][2] = s0 - s1;
    v[q][3] = d0 - d1;
  }
}
// a pair of operands, which the BF16 operator rounds (one conversion for both)
template <bool BF>
__device__ __forceinline__ float2 operands(float x, float y) {
  if constexpr (BF) {
    unsigned p;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p) : "f"(y), "f"(x));  // y in the upper half
    return make_float2(__uint_as_float(p << 16), __uint_as_float(p & 0xffff0000u));
  } else {
    return make_float2(x, y);
  }
}
template <bool BF, int FORM>
__device__ __forceinline__ void face_values(const float* r0, const float* r1, float (&v)[3][4], float (&own)[3]) {
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    own[q] = r0[q];
    const float2 a = operands<BF>(own[q], r0[3 + q]);
    const float2 b = operands<BF>(r1[q], r1[3 + q]);
    float2 p = a, m = b;
    if (FORM == kFaces) {
      p = zbutterfly(add2(a, b));
      m = zbutterfly(sub2(a, b));
      if (q == 2) {
        p = swap2(p);
        m = swap2(m);
      }
    }
    v[q][0] = p.x;
    v[q][1] = p.y;
    v[q][2] = m.x;
    v[q][3] = m.y;
  }
}

// The element between faces p (low x) and c (high x): its contributions lo and hi to
// them, in the faces' representation, scaled by the modulus E.
template <bool DENSE, bool BF, int FORM>
__device__ __forceinline__ void element_faces(const double (&p)[3][4], const double (&c)[3][4], double E,
                                              const double* cw, double (&lo)[3][4], double (&hi)[3][4]) {
  if constexpr (FORM != kFaces) {
    element_product(p, c, E, cw, lo, hi);
  } else {
    double w[3][8], v[3][8];
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        w[q][s] = p[q][s] + c[q][s];
        w[q][4 + s] = p[q][s] - c[q][s];
      }
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const double in[3] = {w[0][b ^ 4], w[1][b ^ 2], w[2][b ^ 1]};
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        double acc = 0.0;
        bool first = true;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          if (!DENSE && !block_entry(b, r, k)) continue;
          const double co = c_wht64[b][3 * r + k];
          acc = first ? co * in[k] : fma(co, in[k], acc);
          first = false;
        }
        v[r][b ^ (4 >> r)] = E * acc;
      }
    }
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        lo[q][s] = v[q][s] + v[q][4 + s];
        hi[q][s] = v[q][s] - v[q][4 + s];
      }
  }
}
template <bool DENSE, bool BF, int FORM>
__device__ __forceinline__ void element_faces(const float (&p)[3][4], const float (&c)[3][4], float E,
                                              const double*, float (&lo)[3][4], float (&hi)[3][4]) {
  float2 a[3][2], b[3][2], l[3][2], h[3][2];
#pragma unroll
  for (int q = 0; q < 3; ++q)
#pragma unroll
    for (int y = 0; y < 2; ++y) {
      a[q][y] = make_float2(p[q][2 * y], p[q][2 * y + 1]);
      b[q][y] = make_float2(c[q][2 * y], c[q][2 * y + 1]);
    }
  if constexpr (FORM == kFaces) {
    float2 w[3][4], v[3][4];
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
      for (int y = 0; y < 2; ++y) {
        w[q][y] = add2(a[q][y], b[q][y]);
        w[q][2 + y] = sub2(a[q][y], b[q][y]);
      }
    blocks2<true, BF>(w, v);
    const float2 E2 = make_float2(E, E);
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
      for (int y = 0; y < 2; ++y) {
        const float2 r = __fmul2_rn(E2, v[q][2 + y]);
        l[q][y] = __ffma2_rn(E2, v[q][y], r);
        h[q][y] = __ffma2_rn(E2, v[q][y], make_float2(-r.x, -r.y));
      }
  } else {
    element_product2(a, b, E, l, h);
  }
#pragma unroll
  for (int q = 0; q < 3; ++q)
#pragma unroll
    for (int y = 0; y < 2; ++y) {
      lo[q][2 * y] = l[q][y].x;
      lo[q][2 * y + 1] = l[q][y].y;
      hi[q][2 * y] = h[q][y].x;
      hi[q][2 * y + 1] = h[q][y].y;
    }
}

// A face's sum t (one component) as its four corners f[2 dy + dz].
template <int FORM>
__device__ __forceinline__ void face_corners(const double (&t)[4], int, double (&f)[4]) {
  if (FORM != kFaces) {
#pragma unroll
    for (int s = 0; s < 4; ++s) f[s] = t[s];
    return;
  }
  const double s0 = t[0] + t[1], d0 = t[0] - t[1], s1 = t[2] + t[3], d1 = t[2] - t[3];
  f[0] = s0 + s1;
  f[1] = d0 + d1;
  f[2] = s0 - s1;
  f[3] = d0 - d1;
}
template <int FORM>
__device__ __forceinline__ void face_corners(const float (&t)[4], int q, float (&f)[4]) {
  float2 a = make_float2(t[0], t[1]), b = make_float2(t[2], t[3]);
  if (FORM == kFaces) {
    if (q == 2) {
      a = swap2(a);
      b = swap2(b);
    }
    const float2 e = zbutterfly(a), o = zbutterfly(b);
    a = add2(e, o);
    b = sub2(e, o);
  }
  f[0] = a.x;
  f[1] = a.y;
  f[2] = b.x;
  f[3] = b.y;
}

// a + b = s + e
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
  s = __fadd_rn(a, b);
  const float t = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t));
}
__device__ __forceinline__ void two_sum(float2 a, float2 b, float2& s, float2& e) {
  s = add2(a, b);
  const float2 t = sub2(s, a);
  e = add2(sub2(a, sub2(s, t)), sub2(b, t));
}
// A node's sum over its four face corners: its own thread's, the z and y neighbours'
// and the diagonal one's.  The element forms keep the order that the solves' bits rest
// on; kFaces adds in pairs, which rounds smaller sums (relative 2-norm against 64 bits,
// FP32 at 512k elements: 6.04e-8, one after the other 6.19e-8, element by element 6.13e-8).
// The BF16 operator also adds what these three additions lose and transforms its faces
// back element by element (sweep_kernel): 4.35e-8, where faces summed first gave 5.31e-8
// and a dense product of the rounded matrix gives 4.56e-8, for 59.7 us at 2M elements
// against 55.6.
template <bool BF, int FORM, typename T>
__device__ __forceinline__ void corner_sums(const T (&own)[3], const T* z, const T* y, const T* yz, T (&ku)[3]) {
  if constexpr (BF) {
    float2 s[3], e[3];  // pairs: (own + y, z + yz)
#pragma unroll
    for (int q = 0; q < 3; ++q) two_sum(make_float2(own[q], z[q]), make_float2(y[q], yz[q]), s[q], e[q]);
    float2 s01, e01;
    two_sum(make_float2(s[0].x, s[1].x), make_float2(s[0].y, s[1].y), s01, e01);
    const float2 l01 = add2(add2(make_float2(e[0].x, e[1].x), make_float2(e[0].y, e[1].y)), e01);
    const float2 k01 = add2(s01, l01);
    ku[0] = k01.x;
    ku[1] = k01.y;
    float s2, e2;
    two_sum(s[2].x, s[2].y, s2, e2);
    ku[2] = add_rn(s2, add_rn(add_rn(e[2].x, e[2].y), e2));
  } else {
#pragma unroll
    for (int q = 0; q < 3; ++q)
      ku[q] = FORM == kFaces ? add_rn(add_rn(own[q], z[q]), add_rn(y[q], yz[q]))
                             : add_rn(add_rn(add_rn(own[q], y[q]), z[q]), yz[q]);
  }
}

// Vectors an epilogue reads per DOF besides the operator's own output and input.
template <int EPI>
constexpr int epi_operands() {
  return EPI == EPI_APPLY ? 0 : (EPI == EPI_RESID ? 1 : (EPI == EPI_CHEB ? 3 : 2));
}

// The epilogues of one node: operands o[0..2] = b, o[3..5] = dinv, o[6..8] = d,
// staged by the thread itself.  off: first DOF of the node, fr its free bits.
template <typename T, int EPI>
__device__ __forceinline__ void node_epilogue(const EpiArgs& ea, int64_t off, unsigned fr, const T* o, const T (&ku)[3],
                                              const T (&x)[3]) {
  T* py = (EPI == EPI_APPLY || EPI == EPI_RESID ? (T*)ea.y : (T*)ea.xo) + off;
  T* pd = (T*)ea.d + off;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const bool f = (fr >> c) & 1;
    T r = T(0), d = T(0);
    if (EPI == EPI_APPLY) {
      r = ku[c];
    } else if (EPI == EPI_RESID) {
      r = sub_rn(o[c], ku[c]);
    } else if (EPI == EPI_CHEB1) {
      d = mul_rn(o[3 + c], sub_rn(o[c], ku[c]));
      r = add_rn(x[c], mul_rn((T)ea.s1, d));
    } else if (EPI == EPI_CHEB) {
      const T z = mul_rn(o[3 + c], sub_rn(o[c], ku[c]));
      d = mul_rn((T)ea.s1, add_rn(z, mul_rn((T)ea.s2, o[6 + c])));
      r = add_rn(x[c], d);
    } else {
      r = add_rn(x[c], mul_rn(mul_rn((T)ea.s1, o[3 + c]), sub_rn(o[c], ku[c])));
    }
    py[c] = f ? r : T(0);
    if (EPI == EPI_CHEB1 || EPI == EPI_CHEB) pd[c] = f ? d : T(0);
  }
}

constexpr int kSweepThreads = 128;  // of a block at most
constexpr int kPlaneBufs = 4;       // node-plane tiles: one being read, two in flight, one just read
constexpr int kTileLoads = 8;       // values of a plane tile staged per thread at most; launch checks

// Blocks of 128 threads resident per SM, as the registers allow without spills:
// three in FP64 (168 registers), four in FP32 (at most 128; five at 96 spilled up to 56
// bytes: 31.7 us for the operator of 1M elements, four 28.3).
template <typename T, bool DENSE, int FORM>
constexpr int sweep_resident() { return sizeof(T) == 8 ? (FORM == kFaces && DENSE ? 2 : 3) : 4; }

// Each block stages its (bj+1) x (bk+1) node tile of one x-plane in shared memory
// with asynchronous copies, one value each, consecutive threads on consecutive
// values of a tile row; values outside the mesh are zeroed once (their set is the
// same for every plane).  The epilogue's operands of a plane come the same way, one
// plane ahead, into slots of the thread's own: read by plain loads they cost an L2
// round trip per plane between the barrier and the update.  Element plane ie couples
// node planes ie and ie + 1; of those only ie + 1 is read (plane ie is still in registers, transformed).  One
// barrier per plane: it makes plane ie + 2 visible (every thread waits for its own
// copies first), frees the buffer of plane ie - 1 and publishes the face sums,
// which alternate between two buffers.
//
// The kernel is bound by latency, not by memory or issue: the grid holds some three
// blocks of three or four warps an SM (512k elements: 16-19 % of the warps, issue in 42 %
// of the cycles in FP64 and 50 % in FP32, reads at the compulsory bytes), and a plane is a chain
// of ~300 instructions a warp around one barrier.  Addresses are running pointers and
// immediate offsets to keep that chain short (the face sums are stored nine to an
// element for that reason: 9 words apart is also free of bank conflicts in both types).
//
// Operator of 1M elements: FP64 87 us before (42 now; its 58 MB at 6.6 TB/s take
// 9), FP32 45 (28); 512k: FP64 50 (31), FP32 24 (20); 2M in FP32 101 (49).  The element
// form of the solves from a cold L2, 512k: FP64 product 39.3 us, FP32 Jacobi step 28.7.
//
// FORM: how an element's product is evaluated.  kFaces transforms a face once for
// two elements, as above.  The products inside a solve -- smoothing steps, residuals
// and the hierarchy's own FP64 operator -- keep the element-by-element evaluation
// instead: FP32 cycles turn a difference of 1e-16 in a Krylov vector into 1e-8 of the
// displacement of nodes that hang in void alone, the nested Krylov solves of the FP64
// stacks into 1e-9 of all of it.  It takes about 1.4 times the arithmetic of kFaces.
//
// COMPACT: u and y are the free-DOF vectors of the C interface, so neither an
// expanded copy of u nor a full result is written.  pinfo[plane] is the free index
// of the first DOF of a node plane that is wholly free -- its values then lie as in
// the full layout --, -1 otherwise; on those planes (supports) ninfo[node] gives 8 *
// (free index of the node's first free DOF) + its three free bits.
template <typename T, int EPI, bool DENSE, bool BF, bool COMPACT, int FORM>
__global__ void __launch_bounds__(kSweepThreads, sweep_resident<T, DENSE, FORM>())
    sweep_kernel(Grid g, SweepShape sh, const T* __restrict__ E, const uint8_t* __restrict__ nmask,
                 const T* __restrict__ u, const int32_t* __restrict__ ninfo,
                 const int32_t* __restrict__ pinfo, EpiArgs ea) {
  if (guard_off(ea.guard)) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int NT = sh.bj * sh.bk;
  const int W = 3 * (sh.bk + 1);           // values per tile row
  const int PV = (sh.bj + 1) * W;          // one plane tile
  constexpr int NO = 3 * epi_operands<EPI>();
  T* F = reinterpret_cast<T*>(smem_raw);   // face sums [2][NT][9]
  T* P = F + 18 * NT;                      // plane tiles [kPlaneBufs][PV]
  T* O = P + kPlaneBufs * PV;              // epilogue operands [2][NT][NO]
  const int t = threadIdx.x;
  __shared__ __align__(16) double cw[sizeof(T) == 8 && FORM != kFaces ? 8 * kBlockCoefs : 2];
  if (sizeof(T) == 8 && FORM != kFaces)
    for (int k = t; k < 8 * kBlockCoefs; k += NT)
      cw[k] = k % kBlockCoefs < 9 ? c_wht64[k / kBlockCoefs][k % kBlockCoefs] : 0.0;
  const int tj = t / sh.bk, tk = t - tj * sh.bk;
  const int nbk = (g.nz + sh.bk - 1) / (sh.bk - 1);  // ceil((nz+1)/(bk-1))
  const int bjI = blockIdx.x / nbk, bkI = blockIdx.x - bjI * nbk;
  const int jb = bjI * (sh.bj - 1) - 1;  // first tile node row = first element row (a halo)
  const int kb = bkI * (sh.bk - 1) - 1;
  const int je = jb + tj, ke = kb + tk;
  const int i0 = blockIdx.y * sh.cx, i1 = min(i0 + sh.cx, g.nx + 1);
  const bool colv = je >= 0 && je < g.ny && ke >= 0 && ke < g.nz;
  const bool own_node = tj >= 1 && tk >= 1 && je <= g.ny && ke <= g.nz;
  const int NZ1 = g.nz + 1, plane_nodes = (g.ny + 1) * NZ1;
  const int last = min(i1, g.nx);  // last node plane read

  // tile values t, t + NT, ...: DOF offset in a plane, the same for every plane
  int rel[kTileLoads];
  unsigned okm = 0;
#pragma unroll
  for (int q = 0; q < kTileLoads; ++q) {
    rel[q] = 0;
    const int v = t + q * NT;
    if (v < PV) {
      const int row = v / W, col = v - row * W;
      const int j = jb + row, k = kb + col / 3;
      if (j >= 0 && j <= g.ny && k >= 0 && k <= g.nz) {
        okm |= 1u << q;
        rel[q] = 3 * (j * NZ1 + kb) + col;
      } else {
#pragma unroll
        for (int p = 0; p < kPlaneBufs; ++p) P[p * PV + v] = T(0);
      }
    }
  }
  // node plane p into its tile buffer; first: pinfo[p] (COMPACT)
  auto issue_plane = [&](int p, int first) {
    T* dst = P + (p & (kPlaneBufs - 1)) * PV + t;
    if (COMPACT && first < 0) {
      const int32_t* info = ninfo + (int64_t)p * plane_nodes;
#pragma unroll
      for (int q = 0; q < kTileLoads; ++q)
        if ((okm >> q) & 1) {
          const int nd = rel[q] / 3, c = rel[q] - 3 * nd, ni = info[nd];
          const bool free_dof = ((ni >> c) & 1) != 0;
          cp_async_elem(dst + q * NT, free_dof ? u + (ni >> 3) + __popc(ni & ((1 << c) - 1)) : u, free_dof);
        }
    } else {
      const T* src = COMPACT ? u + first : u + (int64_t)p * 3 * plane_nodes;
#pragma unroll
      for (int q = 0; q < kTileLoads; ++q)
        if ((okm >> q) & 1) cp_async_elem(dst + q * NT, src + rel[q], true);
    }
  };
  auto plane_first = [&](int p) { return COMPACT && p <= last ? pinfo[p] : 0; };
  // epilogue operands of the thread's node in plane ie (first DOF off)
  auto issue_operands = [&](int ie, int64_t off) {
    if constexpr (NO > 0) {
      if (own_node) {
        T* dst = O + ((ie & 1) * NT + t) * NO;
        const T* src[3] = {(const T*)ea.b + off, (const T*)ea.dinv + off, (const T*)ea.d + off};
#pragma unroll
        for (int k = 0; k < NO; ++k) cp_async_elem(dst + k, src[k / 3] + k % 3, true);
      }
    }
  };

  const int is = max(i0 - 1, 0);  // first element plane (the halo plane below i0, if there is one)
  int64_t node = (int64_t)i0 * plane_nodes + je * NZ1 + ke;
  issue_plane(is, plane_first(is));
  issue_operands(i0, 3 * node);
  cp_async_commit();
#pragma unroll
  for (int d = 1; d <= 2; ++d) {
    if (is + d <= last) issue_plane(is + d, plane_first(is + d));
    cp_async_commit();
  }
  int first_next = plane_first(is + 3);  // of the plane issued next
  const int64_t eplane = (int64_t)g.ny * g.nz;
  const T* Ep = E + (is * eplane + (int64_t)je * g.nz + ke);  // dereferenced only for columns of the mesh
  T En = colv && is < g.nx ? *Ep : T(0);
  // free bits of the thread's next node (COMPACT: pinfo of its plane)
  auto node_bits = [&](int ie, int64_t nd) -> int { return COMPACT ? pinfo[ie] : (own_node ? (int)nmask[nd] : 0); };
  int bits_next = node_bits(i0, node);
  cp_async_wait_all_but_one();
  __syncthreads();
  const int at = tj * W + 3 * tk;
  T p[3][4], carry[3][4], own[3];
  {
    const T* r = P + (is & (kPlaneBufs - 1)) * PV + at;
    face_values<BF, FORM>(r, r + W, p, own);
  }
#pragma unroll
  for (int q = 0; q < 3; ++q)
#pragma unroll
    for (int s = 0; s < 4; ++s) carry[q][s] = T(0);

  for (int ie = is; ie < i1; ++ie) {
    const bool sum = ie >= i0;
    const bool epi = own_node && sum;
    if (ie + 3 <= last) issue_plane(ie + 3, first_next);
    if (COMPACT) first_next = plane_first(ie + 4);
    if (sum && ie + 1 < i1) issue_operands(ie + 1, 3 * (node + plane_nodes));
    cp_async_commit();
    const int bits = bits_next;
    if (sum && ie + 1 < i1) bits_next = node_bits(ie + 1, node + plane_nodes);
    const T Ee = En;
    Ep += eplane;
    En = colv && ie + 1 < g.nx ? *Ep : T(0);
    T tot[3][4], xv[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) xv[q] = own[q];
    if (ie < g.nx) {
      T c[3][4], lo[3][4], hi[3][4];
      const T* r = P + ((ie + 1) & (kPlaneBufs - 1)) * PV + at;
      face_values<BF, FORM>(r, r + W, c, own);
      element_faces<DENSE, BF, FORM>(p, c, Ee, cw, lo, hi);
      if constexpr (BF) {
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          T f[4];
          face_corners<FORM>(lo[q], q, f);
#pragma unroll
          for (int s = 0; s < 4; ++s) lo[q][s] = f[s];
          face_corners<FORM>(hi[q], q, f);
#pragma unroll
          for (int s = 0; s < 4; ++s) hi[q][s] = f[s];
        }
      }
#pragma unroll
      for (int q = 0; q < 3; ++q)
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          tot[q][s] = add_rn(carry[q][s], lo[q][s]);
          carry[q][s] = hi[q][s];
          p[q][s] = c[q][s];
        }
    } else {
#pragma unroll
      for (int q = 0; q < 3; ++q)
#pragma unroll
        for (int s = 0; s < 4; ++s) tot[q][s] = carry[q][s];
    }
    T* buf = F + ((ie & 1) * NT + t) * 9;
    T f0[3];
    if (sum) {
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        T f[4];
        face_corners<BF ? kElement : FORM>(tot[q], q, f);
        f0[q] = f[0];  // corner (0, 0) is the thread's own node
#pragma unroll
        for (int s = 1; s < 4; ++s) buf[3 * (s - 1) + q] = f[s];
      }
    }
    cp_async_wait_all_but_one();
    __syncthreads();
    if (epi) {
      const T* bz = buf - 9;
      const T* by = buf - 9 * sh.bk;
      T ku[3];
      corner_sums<BF, FORM>(f0, bz, by + 3, by + 6 - 9, ku);
      if constexpr (COMPACT) {
        if (bits >= 0) {
          T* py = (T*)ea.y + bits + 3 * (je * NZ1 + ke);
#pragma unroll
          for (int q = 0; q < 3; ++q) py[q] = ku[q];
        } else {
          const int ni = ninfo[node];
          T* py = (T*)ea.y + (ni >> 3);
#pragma unroll
          for (int q = 0; q < 3; ++q)
            if ((ni >> q) & 1) py[__popc(ni & ((1 << q) - 1))] = ku[q];
        }
      } else {
        T o[9];
        const T* src = O + ((ie & 1) * NT + t) * NO;
#pragma unroll
        for (int k = 0; k < NO; ++k) o[k] = src[k];
        node_epilogue<T, EPI>(ea, 3 * node, bits, o, ku, xv);
      }
    }
    if (sum) node += plane_nodes;
  }
}

template <typename T>
static size_t sweep_smem(const SweepShape& sh, int operands) {
  const size_t NT = (size_t)sh.bj * sh.bk, PV = (size_t)(sh.bj + 1) * 3 * (sh.bk + 1);
  return sizeof(T) * ((18 + 6 * operands) * NT + kPlaneBufs * PV);
}

bool fine_shape_ok(DType t, const Grid& g, const SweepShape& sh) {
  const int NT = sh.bj * sh.bk;
  return sh.bk >= 2 && sh.bj >= 2 && sh.cx >= 1 && NT <= kSweepThreads &&
         (sh.bj + 1) * 3 * (sh.bk + 1) <= kTileLoads * NT && div_up(g.nx + 1, sh.cx) <= 65535 &&
         4 * (int64_t)(g.ny + 1) * (g.nz + 1) < (int64_t(1) << 31) &&
         (t == F64 ? sweep_smem<double>(sh, 3) : sweep_smem<float>(sh, 3)) <= 200 * 1024;
}

template <typename T, int EPI, bool DENSE, bool BF, bool COMPACT, int FORM>
static cudaError_t launch_sweep_as(const Grid& g, const SweepShape& sh, const T* E, const uint8_t* nmask, const T* u,
                                   const int32_t* ninfo, const int32_t* pinfo, const EpiArgs& ea, cudaStream_t s) {
  if (!fine_shape_ok(sizeof(T) == 8 ? F64 : F32, g, sh)) return cudaErrorInvalidConfiguration;
  auto kernel = sweep_kernel<T, EPI, DENSE, BF, COMPACT, FORM>;
  static std::atomic<uint64_t> attr_done;
  const cudaError_t ea0 = once_per_device(attr_done, [&] {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  });
  if (ea0 != cudaSuccess) return ea0;
  const int nbj = (g.ny + sh.bj - 1) / (sh.bj - 1);
  const int nbk = (g.nz + sh.bk - 1) / (sh.bk - 1);
  dim3 grid(nbj * nbk, div_up(g.nx + 1, sh.cx));
  kernel<<<grid, sh.bj * sh.bk, sweep_smem<T>(sh, epi_operands<EPI>()), s>>>(g, sh, E, nmask, u, ninfo, pinfo, ea);
  return sf_launched(1);
}

template <typename T, int EPI, bool BF>
static cudaError_t launch_sweep(const Grid& g, const SweepShape& sh, const void* E, const uint8_t* nmask,
                                const void* u, const EpiArgs& ea, cudaStream_t s) {
  if constexpr (sizeof(T) == 8) {
    if ((EPI != EPI_APPLY && EPI != EPI_RESID) || ea.by_element)
      return launch_sweep_as<T, EPI, true, false, false, kElement>(g, sh, (const T*)E, nmask, (const T*)u, nullptr,
                                                                   nullptr, ea, s);
  }
  if constexpr (sizeof(T) == 4 && !BF && EPI != EPI_APPLY) {
    return launch_sweep_as<T, EPI, true, false, false, kElement>(g, sh, (const T*)E, nmask, (const T*)u, nullptr,
                                                                 nullptr, ea, s);
  } else if constexpr (sizeof(T) == 4) {
    return launch_sweep_as<T, EPI, true, BF, false, kFaces>(g, sh, (const T*)E, nmask, (const T*)u, nullptr, nullptr,
                                                            ea, s);
  } else if constexpr (EPI == EPI_APPLY || EPI == EPI_RESID) {
    return pattern_on_device()
               ? launch_sweep_as<T, EPI, false, BF, false, kFaces>(g, sh, (const T*)E, nmask, (const T*)u, nullptr,
                                                                   nullptr, ea, s)
               : launch_sweep_as<T, EPI, true, BF, false, kFaces>(g, sh, (const T*)E, nmask, (const T*)u, nullptr,
                                                                  nullptr, ea, s);
  }
  return cudaErrorInvalidValue;
}

template <typename T, bool BF>
static cudaError_t launch_sweep_epi(Epi epi, const Grid& g, const SweepShape& sh, const void* E, const uint8_t* nmask,
                                    const void* u, const EpiArgs& ea, cudaStream_t s) {
  switch (epi) {
    case EPI_APPLY: return launch_sweep<T, EPI_APPLY, BF>(g, sh, E, nmask, u, ea, s);
    case EPI_RESID: return launch_sweep<T, EPI_RESID, BF>(g, sh, E, nmask, u, ea, s);
    case EPI_CHEB1: return launch_sweep<T, EPI_CHEB1, BF>(g, sh, E, nmask, u, ea, s);
    case EPI_CHEB: return launch_sweep<T, EPI_CHEB, BF>(g, sh, E, nmask, u, ea, s);
    case EPI_JAC: return launch_sweep<T, EPI_JAC, BF>(g, sh, E, nmask, u, ea, s);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_fine(DType t, Epi epi, const Grid& g, const SweepShape& sh, const void* E,
                        const uint8_t* nmask, const void* u, const EpiArgs& ea, cudaStream_t s) {
  if (t == F64) return launch_sweep_epi<double, false>(epi, g, sh, E, nmask, u, ea, s);
  if (t == F32) return launch_sweep_epi<float, false>(epi, g, sh, E, nmask, u, ea, s);
  // BF16 operands (u and KE rounded to bf16), FP32 accumulation and FP32 vectors
  if (t == BF16) return launch_sweep_epi<float, true>(epi, g, sh, E, nmask, u, ea, s);
  return cudaErrorInvalidValue;
}

cudaError_t launch_fine_compact(const Grid& g, const SweepShape& sh, const double* E, const int32_t* ninfo,
                                const int32_t* pinfo, const double* u_free, double* y_free, cudaStream_t s) {
  EpiArgs ea;
  ea.y = y_free;
  return pattern_on_device()
             ? launch_sweep_as<double, EPI_APPLY, false, false, true, kFaces>(g, sh, E, nullptr, u_free, ninfo, pinfo, ea, s)
             : launch_sweep_as<double, EPI_APPLY, true, false, true, kFaces>(g, sh, E, nullptr, u_free, ninfo, pinfo, ea, s);
}

// ----------------------------------------------------------------------------
// diag(K_ff): per node, sum over the adjacent elements of E_e * KE_jj
// (MatrixFreeKff.extract_diagonal, gpu_fem/solver_v2.py:1228-1251).
__global__ void fine_diag_kernel(Grid g, const double* __restrict__ E, const uint8_t* __restrict__ mask,
                                 double* __restrict__ diag) {
  const int64_t node = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (node >= g.nn) return;
  const int NZ = g.nz + 1, NY = g.ny + 1;
  const int k = (int)(node % NZ);
  const int j = (int)((node / NZ) % NY);
  const int i = (int)(node / ((int64_t)NZ * NY));
  double acc[3] = {0.0, 0.0, 0.0};
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    // element whose corner q sits on this node
    const int dx = q >> 2, dy = (q >> 1) & 1, dz = q & 1;
    const int ei = i - dx, ej = j - dy, ek = k - dz;
    if (ei < 0 || ej < 0 || ek < 0 || ei >= g.nx || ej >= g.ny || ek >= g.nz) continue;
    const double Ee = E[((int64_t)ei * g.ny + ej) * g.nz + ek];
#pragma unroll
    for (int c = 0; c < 3; ++c) acc[c] += Ee * c_kediag[q * 3 + c];
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) diag[3 * node + c] = mask[3 * node + c] ? acc[c] : 0.0;
}

cudaError_t launch_fine_diag(const Grid& g, const double* E, const uint8_t* mask, double /*kd*/,
                             double* diag, cudaStream_t s) {
  fine_diag_kernel<<<div_up(g.nn, 256), 256, 0, s>>>(g, E, mask, diag);
  return sf_launched(1);
}

// ----------------------------------------------------------------------------
// 3x3 node-block Jacobi (NodeBlockJacobiMF, gpu_fem/solver_v2.py:1268-1451):
// block(n) = sum_e E_e * KE[node block of n in e]; all-free nodes store the
// block inverse, partially constrained nodes store 1/diag for their free
// components (the reference's scalar fallback), constrained components 0.
__global__ void node_blocks_kernel(Grid g, const double* __restrict__ E, const uint8_t* __restrict__ mask,
                                   const double* __restrict__ diag_full, double* __restrict__ binv) {
  const int64_t node = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (node >= g.nn) return;
  const int NZ = g.nz + 1, NY = g.ny + 1;
  const int k = (int)(node % NZ);
  const int j = (int)((node / NZ) % NY);
  const int i = (int)(node / ((int64_t)NZ * NY));
  double B[9];
#pragma unroll
  for (int r = 0; r < 9; ++r) B[r] = 0.0;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int dx = q >> 2, dy = (q >> 1) & 1, dz = q & 1;
    const int ei = i - dx, ej = j - dy, ek = k - dz;
    if (ei < 0 || ej < 0 || ek < 0 || ei >= g.nx || ej >= g.ny || ek >= g.nz) continue;
    const double Ee = E[((int64_t)ei * g.ny + ej) * g.nz + ek];
#pragma unroll
    for (int r = 0; r < 9; ++r) B[r] += Ee * c_kenb[q][r];
  }
  const bool f0 = mask[3 * node], f1 = mask[3 * node + 1], f2 = mask[3 * node + 2];
  double out[9];
#pragma unroll
  for (int r = 0; r < 9; ++r) out[r] = 0.0;
  if (f0 && f1 && f2) {
    const double c00 = B[4] * B[8] - B[5] * B[7];
    const double c01 = B[5] * B[6] - B[3] * B[8];
    const double c02 = B[3] * B[7] - B[4] * B[6];
    const double det = B[0] * c00 + B[1] * c01 + B[2] * c02;
    const double id = 1.0 / det;
    out[0] = c00 * id;
    out[1] = (B[2] * B[7] - B[1] * B[8]) * id;
    out[2] = (B[1] * B[5] - B[2] * B[4]) * id;
    out[3] = c01 * id;
    out[4] = (B[0] * B[8] - B[2] * B[6]) * id;
    out[5] = (B[2] * B[3] - B[0] * B[5]) * id;
    out[6] = c02 * id;
    out[7] = (B[1] * B[6] - B[0] * B[7]) * id;
    out[8] = (B[0] * B[4] - B[1] * B[3]) * id;
  } else {
    const bool fr[3] = {f0, f1, f2};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      // without a scalar diagonal the reference leaves these components at 0
      if (fr[c] && diag_full != nullptr) {
        double d = diag_full[3 * node + c];
        d = fabs(d) > 1e-12 ? d : 1.0;
        out[c * 4] = 1.0 / d;
      }
    }
  }
#pragma unroll
  for (int r = 0; r < 9; ++r) binv[9 * node + r] = out[r];
}

cudaError_t launch_node_blocks(const Grid& g, const double* E, const uint8_t* mask,
                               const double* diag_full, double* binv, cudaStream_t s) {
  node_blocks_kernel<<<div_up(g.nn, 256), 256, 0, s>>>(g, E, mask, diag_full, binv);
  return sf_launched(1);
}

__global__ void node_block_apply_kernel(int64_t nn, const double* __restrict__ binv,
                                        const double* __restrict__ r, double* __restrict__ z,
                                        const int* guard) {
  if (guard_off(guard)) return;
  const int64_t node = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (node >= nn) return;
  const double r0 = r[3 * node], r1 = r[3 * node + 1], r2 = r[3 * node + 2];
  const double* B = binv + 9 * node;
#pragma unroll
  for (int c = 0; c < 3; ++c) z[3 * node + c] = B[3 * c] * r0 + B[3 * c + 1] * r1 + B[3 * c + 2] * r2;
}

cudaError_t launch_node_block_apply(const Grid& g, const double* binv, const double* r, double* z,
                                    const int* guard, cudaStream_t s) {
  node_block_apply_kernel<<<div_up(g.nn, 256), 256, 0, s>>>(g.nn, binv, r, z, guard);
  return sf_launched(1);
}

// ----------------------------------------------------------------------------
// Element strain energy u_e^T KE u_e (SolverV4 sensitivity, gpu_fem/solver_v4.py:257-264).
__global__ void element_energy_kernel(Grid g, const double* __restrict__ u, double* __restrict__ ce) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= g.ne()) return;
  const int ek = (int)(e % g.nz);
  const int ej = (int)((e / g.nz) % g.ny);
  const int ei = (int)(e / ((int64_t)g.nz * g.ny));
  double ue[8][3];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int dx = q >> 2, dy = (q >> 1) & 1, dz = q & 1;
    const int64_t node = ((int64_t)(ei + dx) * (g.ny + 1) + (ej + dy)) * (g.nz + 1) + (ek + dz);
#pragma unroll
    for (int c = 0; c < 3; ++c) ue[q][c] = u[3 * node + c];
  }
  double f[8][3];
  elem_wht(ue, f);
  double acc = 0.0;
#pragma unroll
  for (int q = 0; q < 8; ++q)
#pragma unroll
    for (int c = 0; c < 3; ++c) acc += f[q][c] * ue[q][c];
  ce[e] = acc;
}

cudaError_t launch_element_energy(const Grid& g, const double* u_full, double* ce, cudaStream_t s) {
  element_energy_kernel<<<div_up(g.ne(), 256), 256, 0, s>>>(g, u_full, ce);
  return sf_launched(1);
}

}  // namespace simpfem
