// Learned floor proposer: a small 3D CNN, forward, backward and Adam on the GPU.
// No counterpart in the reference.
//
//   x (N, 1, 16^3) -- the density average-pooled to 16^3 (pool16_kernel)
//   conv 1->16  s1 -> 16^3, conv 16->16 s2 -> 8^3, conv 16->32 s2 -> 4^3,
//   conv 32->32 s2 -> 2^3   (3x3x3, pad 1, ReLU after each)
//   mean over 8 positions (32) ++ 2 probe features -> dense 34 -> 3 -> softmax
//
// Weights are stored and read as bfloat16, biases and every activation and
// accumulation in float32; the float32 master copy is what Adam updates (the
// gradient is taken with respect to the bfloat16 weights).  Parameter layout:
// W1 b1 W2 b2 W3 b3 W4 b4 Wfc bfc, weights [cout][cin][kz][ky][kx].
// Every reduction (weight and bias gradients, the loss) runs in a fixed order,
// so a training run is bitwise reproducible.
//
// The work is 6.4 M multiply-adds a sample forward and twice that backward, all
// on FP32 operands (activations and gradients stay FP32, so the tensor cores'
// narrower inputs are not used); what decides the time is how often an operand is
// read.  The kernels this replaces gave a thread one output value or a block one
// parameter, i.e. two loads per multiply-add: 10.3 ms for a training step of 128
// (weight gradients 4.9, data gradients 4.7, forward 0.7).  Here each layer
// stages its operands in shared memory and a thread keeps a tile of accumulators
// in registers:
//   forward         1-2 channels x 1-2 positions a thread (first layer: 16 x 2)
//   data gradient   2 x 2 x 2 input cells (every parity class of the stride: 27 taps per cell),
//                   two cells x 2-4 input channels a thread
//   weight gradient 4 output channels x 27 taps of one input channel a thread, each thread
//                   one residue of (sample, position) modulo 256, then a tree over the 256
// Sums keep one order whatever the batch: channels, then taps, for the data; for a
// weight 256 interleaved chains and their tree.  A unit within a rounding of its
// ReLU's kink then takes the same side, which a reordered sum would not promise.
// Training step of 128: 10.3 -> 0.46 ms on the device (weight gradients 0.20,
// data gradients 0.12, forward 0.10); one forward of one sample 121 -> 35 us.
#include <math.h>

#include <algorithm>
#include <cstring>

#include "common.cuh"
#include "gmg_impl.h"
#include "simpfem.h"

namespace simpfem {
namespace {

constexpr int kS0 = 16, kVox = kS0 * kS0 * kS0, kFeat = 2, kClass = 3;
constexpr int cin(int l) { return l == 0 ? 1 : (l < 3 ? 16 : 32); }
constexpr int cout(int l) { return l < 2 ? 16 : 32; }
constexpr int sout(int l) { return 16 >> l; }
constexpr int kHidden = 32, kZ = kHidden + kFeat;

// offsets of the parameters: weights and biases of convolution l (l = 4: the dense layer)
constexpr int w_off(int l) { return l == 0 ? 0 : w_off(l - 1) + cout(l - 1) * (cin(l - 1) * 27 + 1); }
constexpr int b_off(int l) { return l < 4 ? w_off(l) + cout(l) * cin(l) * 27 : w_off(4) + kClass * kZ; }
constexpr int kParams = b_off(4) + kClass;
static_assert(kParams == 49017, "parameter count");

constexpr int kTap = 28;  // 27 taps of a channel pair padded to a multiple of 16 bytes

// weights rounded to bfloat16 (values kept in FP32) in the two layouts the
// kernels stage from: wf[ci][tap][co] (forward) and wb[co][ci][kTap] (data gradient)
constexpr int f_off(int l) { return l == 0 ? 0 : f_off(l - 1) + cin(l - 1) * 27 * cout(l - 1); }
constexpr int t_off(int l) { return l < 2 ? 0 : t_off(l - 1) + cout(l - 1) * cin(l - 1) * kTap; }
constexpr int kFwdPad = (f_off(4) + kClass * kZ + 3) / 4 * 4, kBwdWords = t_off(4);
static_assert(f_off(1) % 4 == 0 && f_off(2) % 4 == 0 && f_off(3) % 4 == 0 && t_off(2) % 4 == 0 && t_off(3) % 4 == 0,
              "16-byte starts");

__global__ void pack_weights_kernel(const float* __restrict__ theta, float* __restrict__ wf, float* __restrict__ wb) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kParams) return;
  const float v = __bfloat162float(__float2bfloat16_rn(theta[i]));
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    const int e = i - w_off(l);
    if (e >= 0 && e < cout(l) * cin(l) * 27) {
      const int k = e % 27, ci = (e / 27) % cin(l), co = e / (27 * cin(l));
      wf[f_off(l) + (ci * 27 + k) * cout(l) + co] = v;
      if (l > 0) wb[t_off(l) + (co * cin(l) + ci) * kTap + k] = v;
    }
  }
  const int e = i - w_off(4);
  if (e >= 0 && e < kClass * kZ) wf[f_off(4) + e] = v;
}

__device__ __forceinline__ void copy_f4(float* dst, const float* __restrict__ src, int n, int tid, int nt) {
  for (int e = 4 * tid; e < n; e += 4 * nt)
    *reinterpret_cast<float4*>(dst + e) = *reinterpret_cast<const float4*>(src + e);
}

// ---- first layer: 1 -> 16 channels, stride 1.  A block makes one plane of one
// sample; a thread two x-adjacent positions of all 16 channels.
constexpr int kC0Threads = 128;
__global__ void __launch_bounds__(kC0Threads) conv0_fwd_kernel(const float* __restrict__ x, const float* __restrict__ wf,
                                                               const float* __restrict__ bias, float* __restrict__ y) {
  __shared__ __align__(16) float ws[27 * 16];
  __shared__ float in[3][18][18];
  const int n = blockIdx.x >> 4, oz = blockIdx.x & 15, tid = threadIdx.x;
  copy_f4(ws, wf + f_off(0), 27 * 16, tid, kC0Threads);
  for (int e = tid; e < 3 * 18 * 18; e += kC0Threads) {
    const int c = e % 18, r = (e / 18) % 18, p = e / 324;
    const int iz = oz + p - 1, iy = r - 1, ix = c - 1;
    const bool ok = iz >= 0 && iz < 16 && iy >= 0 && iy < 16 && ix >= 0 && ix < 16;
    in[p][r][c] = ok ? x[((int64_t)n << 12) + (iz * 16 + iy) * 16 + ix] : 0.f;
  }
  __syncthreads();
  const int oy = tid >> 3, ox = (tid & 7) * 2;
  float acc[16][2];
#pragma unroll
  for (int c = 0; c < 16; ++c) acc[c][0] = acc[c][1] = bias[c];
#pragma unroll
  for (int kz = 0; kz < 3; ++kz)
#pragma unroll
    for (int ky = 0; ky < 3; ++ky) {
      float v[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) v[t] = in[kz][oy + ky][ox + t];
#pragma unroll
      for (int kx = 0; kx < 3; ++kx) {
        const float4* w4 = reinterpret_cast<const float4*>(ws + ((kz * 3 + ky) * 3 + kx) * 16);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float4 w = w4[q];
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            acc[4 * q][t] = fmaf(w.x, v[kx + t], acc[4 * q][t]);
            acc[4 * q + 1][t] = fmaf(w.y, v[kx + t], acc[4 * q + 1][t]);
            acc[4 * q + 2][t] = fmaf(w.z, v[kx + t], acc[4 * q + 2][t]);
            acc[4 * q + 3][t] = fmaf(w.w, v[kx + t], acc[4 * q + 3][t]);
          }
        }
      }
    }
#pragma unroll
  for (int c = 0; c < 16; ++c)
    *reinterpret_cast<float2*>(y + (((int64_t)n * 16 + c) << 12) + (oz * 16 + oy) * 16 + ox) =
        make_float2(fmaxf(acc[c][0], 0.f), fmaxf(acc[c][1], 0.f));
}

// ---- stride-2 layers.  Shapes of layer l: CI channels of S^3 -> CO of (S/2)^3.
// Input planes are staged with one zero plane, row and column before them (the
// only padding a stride-2 window over an even extent reaches).
template <int CI, int CO, int S, int COB, int OZB, int CT, int PX>
struct ConvS2 {
  static constexpr int O = S / 2, P = S + 1, PL = 2 * (OZB - 1) + 3;  // staged planes
  static constexpr int POS = OZB * O * O, TP = POS / PX, TC = COB / CT;
  static constexpr int THREADS = TP * TC, BLOCKS = O / OZB * (CO / COB);  // per sample
  static constexpr int IN = (CI * PL * P * P + 3) / 4 * 4, W = CI * 27 * COB;
  static constexpr size_t SMEM = sizeof(float) * (IN + W);
};

// Rows are read as float4, four of them in flight per thread.  Planes before the
// first are zero, as are the padding plane's row and column.
template <int CI, int S, int PL, int NT>
__device__ __forceinline__ void stage_planes(float* dst, const float* __restrict__ xn, int iz0, int tid) {
  constexpr int P = S + 1, V = S / 4, N4 = CI * PL * S * V;
#pragma unroll 4
  for (int e = tid; e < N4; e += NT) {
    const int c = e % V, r = (e / V) % S, p = (e / (V * S)) % PL, ci = e / (V * S * PL);
    const int iz = iz0 + p;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (iz >= 0) v = *reinterpret_cast<const float4*>(xn + ((ci * S + iz) * S + r) * S + 4 * c);
    float* d = dst + ((ci * PL + p) * P + r + 1) * P + 4 * c + 1;
    d[0] = v.x;
    d[1] = v.y;
    d[2] = v.z;
    d[3] = v.w;
  }
  for (int e = tid; e < CI * PL * P; e += NT) {
    const int q = e % P, pc = e / P;
    dst[pc * P * P + q] = 0.f;
    dst[(pc * P + q) * P] = 0.f;
  }
}

// A block makes OZB output planes of COB channels of one sample, a thread CT
// channels of PX neighbouring positions.
template <int CI, int CO, int S, int COB, int OZB, int CT, int PX>
__global__ void __launch_bounds__(ConvS2<CI, CO, S, COB, OZB, CT, PX>::THREADS)
    conv_s2_fwd_kernel(const float* __restrict__ x, const float* __restrict__ wf, const float* __restrict__ bias,
                       float* __restrict__ y) {
  using C = ConvS2<CI, CO, S, COB, OZB, CT, PX>;
  extern __shared__ __align__(16) float sm[];
  float* in = sm;
  float* ws = sm + C::IN;
  constexpr int ZB = C::O / OZB;
  const int n = blockIdx.x / C::BLOCKS, part = blockIdx.x % C::BLOCKS, tid = threadIdx.x;
  const int oz0 = (part % ZB) * OZB, co0 = (part / ZB) * COB;
#pragma unroll 4
  for (int e = tid; e < C::W / 4; e += C::THREADS) {
    const int q = e % (COB / 4), row = e / (COB / 4);
    reinterpret_cast<float4*>(ws)[e] = *reinterpret_cast<const float4*>(wf + row * CO + co0 + 4 * q);
  }
  stage_planes<CI, S, C::PL, C::THREADS>(in, x + (int64_t)n * CI * S * S * S, 2 * oz0 - 1, tid);
  __syncthreads();
  const int cq = tid % C::TC, pg = tid / C::TC;
  constexpr int GX = C::O / PX;
  const int ox = (pg % GX) * PX, oy = (pg / GX) % C::O, oz = pg / (GX * C::O);
  float acc[CT][PX];
#pragma unroll
  for (int c = 0; c < CT; ++c)
#pragma unroll
    for (int q = 0; q < PX; ++q) acc[c][q] = bias[co0 + CT * cq + c];
#pragma unroll 2
  for (int ci = 0; ci < CI; ++ci) {
    const float* base = in + ((ci * C::PL + 2 * oz) * C::P + 2 * oy) * C::P + 2 * ox;
    const float* wb = ws + ci * 27 * COB + CT * cq;
#pragma unroll
    for (int kz = 0; kz < 3; ++kz)
#pragma unroll
      for (int ky = 0; ky < 3; ++ky) {
        float v[2 * PX + 1];
#pragma unroll
        for (int q = 0; q < 2 * PX + 1; ++q) v[q] = base[(kz * C::P + ky) * C::P + q];
#pragma unroll
        for (int kx = 0; kx < 3; ++kx) {
          float w[CT];
          if (CT == 2) {
            const float2 w2 = *reinterpret_cast<const float2*>(wb + ((kz * 3 + ky) * 3 + kx) * COB);
            w[0] = w2.x;
            w[CT - 1] = w2.y;
          } else {
            w[0] = wb[((kz * 3 + ky) * 3 + kx) * COB];
          }
#pragma unroll
          for (int c = 0; c < CT; ++c)
#pragma unroll
            for (int q = 0; q < PX; ++q) acc[c][q] = fmaf(w[c], v[2 * q + kx], acc[c][q]);
        }
      }
  }
#pragma unroll
  for (int c = 0; c < CT; ++c) {
    float* o = y + ((int64_t)n * CO + co0 + CT * cq + c) * C::O * C::O * C::O + ((oz0 + oz) * C::O + oy) * C::O + ox;
#pragma unroll
    for (int q = 0; q < PX; ++q) o[q] = fmaxf(acc[c][q], 0.f);
  }
}

// Data gradient: dx = conv^T(dy), masked by the input's own ReLU (act > 0); dy
// arrives masked.  Along an axis input 2I takes tap 1 of output I and input
// 2I + 1 takes tap 0 of output I + 1 and tap 2 of output I, so the 27 taps serve
// the 8 inputs of cell (I, J, K) once each.
template <int CI, int CO, int S, int CT, int SPB, int CPART>
struct DgradS2 {
  static constexpr int O = S / 2, P = O + 1;
  static constexpr int TX = O / 2, TCELL = O * O * TX, CIB = CI / CPART, TG = CIB / CT;
  static constexpr int TPS = TCELL * TG, THREADS = TPS * SPB;
  static constexpr int DY = CO * P * P * P;
  static constexpr size_t SMEM = sizeof(float) * ((size_t)CO * CIB * kTap + (size_t)SPB * DY);
};

template <int CI, int CO, int S, int CT, int SPB, int CPART>
__global__ void __launch_bounds__(DgradS2<CI, CO, S, CT, SPB, CPART>::THREADS)
    conv_s2_bwd_data_kernel(int N, const float* __restrict__ dy, const float* __restrict__ wb,
                            const float* __restrict__ act, float* __restrict__ dx) {
  using C = DgradS2<CI, CO, S, CT, SPB, CPART>;
  extern __shared__ __align__(16) float sm[];
  float* ws = sm;                              // [CO][CIB][kTap]
  float* ds = sm + CO * C::CIB * kTap;         // [SPB][CO][P][P][P], zero past the last output
  const int tid = threadIdx.x, n0 = blockIdx.x * SPB, c0 = blockIdx.y * C::CIB;
  for (int e = 4 * tid; e < CO * C::CIB * kTap; e += 4 * C::THREADS) {
    const int co = e / (C::CIB * kTap), r = e % (C::CIB * kTap);
    *reinterpret_cast<float4*>(ws + e) = *reinterpret_cast<const float4*>(wb + (co * CI + c0) * kTap + r);
  }
  for (int e = tid; e < SPB * C::DY; e += C::THREADS) {
    const int c = e % C::P, r = (e / C::P) % C::P, p = (e / (C::P * C::P)) % C::P, nc = e / (C::P * C::P * C::P);
    const bool ok = c < C::O && r < C::O && p < C::O && n0 + nc / CO < N;
    ds[e] = ok ? dy[(((int64_t)n0 * CO + nc) * C::O + p) * C::O * C::O + r * C::O + c] : 0.f;
  }
  __syncthreads();
  const int sp = tid / C::TPS, t = tid % C::TPS, g = t / C::TCELL, cell = t % C::TCELL;
  const int n = n0 + sp;
  const int X = (cell % C::TX) * 2, Y = (cell / C::TX) % C::O, Z = cell / (C::TX * C::O);
  float acc[CT][2][2][4];
#pragma unroll
  for (int c = 0; c < CT; ++c)
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[c][a][b][q] = 0.f;
  for (int co = 0; co < CO; ++co) {
    const float* d = ds + (sp * CO + co) * C::P * C::P * C::P + (Z * C::P + Y) * C::P + X;
    float v[2][2][3];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int q = 0; q < 3; ++q) v[a][b][q] = d[(a * C::P + b) * C::P + q];
#pragma unroll
    for (int c = 0; c < CT; ++c) {
      const float4* w4 = reinterpret_cast<const float4*>(ws + (co * C::CIB + g * CT + c) * kTap);
      float w[kTap];
#pragma unroll
      for (int q = 0; q < kTap / 4; ++q) {
        const float4 f = w4[q];
        w[4 * q] = f.x;
        w[4 * q + 1] = f.y;
        w[4 * q + 2] = f.z;
        w[4 * q + 3] = f.w;
      }
#pragma unroll
      for (int kz = 0; kz < 3; ++kz)
#pragma unroll
        for (int ky = 0; ky < 3; ++ky)
#pragma unroll
          for (int kx = 0; kx < 3; ++kx) {
            const float wk = w[(kz * 3 + ky) * 3 + kx];
            const int pz = kz == 1 ? 0 : 1, py = ky == 1 ? 0 : 1, px = kx == 1 ? 0 : 1;
            const int oz = kz == 0 ? 1 : 0, oy = ky == 0 ? 1 : 0, ox = kx == 0 ? 1 : 0;
            acc[c][pz][py][px] = fmaf(wk, v[oz][oy][ox], acc[c][pz][py][px]);
            acc[c][pz][py][2 + px] = fmaf(wk, v[oz][oy][ox + 1], acc[c][pz][py][2 + px]);
          }
    }
  }
  if (n >= N) return;
#pragma unroll
  for (int c = 0; c < CT; ++c)
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        const int64_t o =
            (((int64_t)n * CI + c0 + g * CT + c) * S + 2 * Z + a) * S * S + (2 * Y + b) * S + 2 * X;
        const float4 m = *reinterpret_cast<const float4*>(act + o);
        const float* r = acc[c][a][b];
        *reinterpret_cast<float4*>(dx + o) = make_float4(m.x > 0.f ? r[0] : 0.f, m.y > 0.f ? r[1] : 0.f,
                                                         m.z > 0.f ? r[2] : 0.f, m.w > 0.f ? r[3] : 0.f);
      }
}

// Sum over the 256 threads of a block of NV values each, as the tree
// v[t] += v[t + w], w = 128 .. 1; valid in thread 0.  buf: 128 * NV floats.
template <int NV>
__device__ __forceinline__ void block_tree_256(float (&v)[NV], float* buf) {
  const int t = threadIdx.x;
#pragma unroll
  for (int w = 128; w >= 32; w >>= 1) {
    __syncthreads();
    if (t >= w && t < 2 * w) {
#pragma unroll
      for (int k = 0; k < NV; ++k) buf[k * w + t - w] = v[k];
    }
    __syncthreads();
    if (t < w) {
#pragma unroll
      for (int k = 0; k < NV; ++k) v[k] += buf[k * w + t];
    }
  }
  if (t < 32) {
#pragma unroll
    for (int k = 0; k < NV; ++k)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
  }
}

// 16 bytes global -> shared, asynchronously; zeros when ok is false (src is then
// any valid address)
__device__ __forceinline__ void cp16(float* dst, const float* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(ok ? 16 : 0));
}
// the same from a source that is aligned to its type only
__device__ __forceinline__ void cp16_by_float(float* dst, const float* src) {
#pragma unroll
  for (int k = 0; k < 4; ++k)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst + k)),
                 "l"(src + k));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int LEFT>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(LEFT));
}
constexpr int kRing = 4;  // steps of samples staged or in flight

// Weight and bias gradients of a stride-2 layer: a block takes 4 output channels of
// one input channel; thread t adds the (sample, position) pairs q = t, t + 256, ...
// in order, 27 taps x 4 channels (and, in the blocks of input channel 0, the
// biases) in registers.  A chain is 2 N / 256 positions long and cannot be split
// over blocks without another order of sums, so a block walks all samples: its
// steps stream through a ring of four asynchronous copies (with one step ahead in
// registers a step waited on the loads: 168 us at batch 128 in the second layer).
// RS: row stride, chosen so that a warp's 64-bit reads of the stride-2 window meet
// each bank once.
template <int CI, int CO, int S, int RS>
struct WgradS2 {
  static constexpr int O = S / 2, P = S + 1, O3 = O * O * O, S3 = S * S * S;
  static constexpr int M = O3 >= 256 ? O3 / 256 : 1, SPI = O3 >= 256 ? 1 : 256 / O3;  // positions a thread, samples a step
  static constexpr int TILE = SPI * P * P * RS, DY = SPI * 4 * O3, STEP = TILE + DY;
  static constexpr int NV = 112, RED = 128 * NV;
  static constexpr size_t SMEM = sizeof(float) * (kRing * STEP > RED ? kRing * STEP : RED);
  static_assert(RS % 4 == 0 && RS >= S, "16-byte rows");
};

template <int CI, int CO, int S, int RS>
__global__ void __launch_bounds__(256, 1) conv_s2_bwd_param_kernel(int N, const float* __restrict__ dy,
                                                                   const float* __restrict__ x,
                                                                   float* __restrict__ gW, float* __restrict__ gb) {
  using C = WgradS2<CI, CO, S, RS>;
  constexpr int P = C::P, O = C::O, V = S / 4;
  extern __shared__ __align__(16) float sm[];
  const int tid = threadIdx.x, ci = blockIdx.x % CI, cq = blockIdx.x / CI;
  // plane 0 and row 0 of a tile stay zero (the padding before the first input)
  for (int e = tid; e < kRing * C::STEP; e += 256) sm[e] = 0.f;
  __syncthreads();
  auto stage = [&](int slot, int n0) {
    float* t = sm + slot * C::STEP;
#pragma unroll
    for (int u = 0; u < C::SPI * C::S3 / 4 / 256; ++u) {
      const int e = tid + 256 * u, sp = e / (C::S3 / 4), r = e % (C::S3 / 4);
      const int c = 4 * (r % V), ry = (r / V) % S, rz = r / (V * S);
      const bool ok = n0 + sp < N;
      cp16(t + ((sp * P + rz + 1) * P + ry + 1) * RS + c,
           x + ((int64_t)(ok ? n0 + sp : 0) * CI + ci) * C::S3 + 4 * r, ok);
    }
#pragma unroll
    for (int u = 0; u < C::DY / 4 / 256; ++u) {
      const int e = tid + 256 * u, sp = e / C::O3, r = e % C::O3;  // O3 float4 a sample: [4][O3 / 4]
      const bool ok = n0 + sp < N;
      cp16(t + C::TILE + sp * 4 * C::O3 + 4 * r, dy + ((int64_t)(ok ? n0 + sp : 0) * CO + 4 * cq) * C::O3 + 4 * r, ok);
    }
  };
  float acc[C::NV];  // [4][27], then the 4 biases
#pragma unroll
  for (int k = 0; k < C::NV; ++k) acc[k] = 0.f;
#pragma unroll
  for (int p = 0; p < kRing - 1; ++p) {
    if (p * C::SPI < N) stage(p, p * C::SPI);
    cp_commit();
  }
  int slot = 0;
  for (int n0 = 0; n0 < N; n0 += C::SPI) {
    cp_wait<kRing - 2>();
    __syncthreads();  // this step's copies are in; the slot of the step before is free
    const int ahead = n0 + (kRing - 1) * C::SPI;
    if (ahead < N) stage((slot + kRing - 1) % kRing, ahead);
    cp_commit();
    const float* t = sm + slot * C::STEP;
#pragma unroll
    for (int m = 0; m < C::M; ++m) {
      const int q = tid + 256 * m, sp = C::SPI > 1 ? q / C::O3 : 0, o = q % C::O3;
      const int ox = o % O, oy = (o / O) % O, oz = o / (O * O);
      const float* b = t + ((sp * P + 2 * oz) * P + 2 * oy) * RS + 2 * ox;
      float d[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) d[c] = t[C::TILE + (sp * 4 + c) * C::O3 + o];
      const int left = ox > 0 ? -1 : 0;
#pragma unroll
      for (int r = 0; r < 9; ++r) {
        const float* row = b + ((r / 3) * P + r % 3) * RS;
        const float2 mid = *reinterpret_cast<const float2*>(row);
        const float lo = row[left];
        const float w[3] = {ox > 0 ? lo : 0.f, mid.x, mid.y};
#pragma unroll
        for (int kx = 0; kx < 3; ++kx)
#pragma unroll
          for (int c = 0; c < 4; ++c) acc[c * 27 + r * 3 + kx] = fmaf(d[c], w[kx], acc[c * 27 + r * 3 + kx]);
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[108 + c] += d[c];
    }
    slot = (slot + 1) % kRing;
  }
  cp_wait<0>();
  block_tree_256<C::NV>(acc, sm);
  if (tid == 0) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
#pragma unroll
      for (int k = 0; k < 27; ++k) gW[((4 * cq + c) * CI + ci) * 27 + k] = acc[c * 27 + k];
      if (ci == 0) gb[4 * cq + c] = acc[108 + c];
    }
  }
}

// First layer's weight and bias gradients, in the same order of sums: a block takes
// one output channel and one row ky of taps, thread t the position (y, x) of every
// plane (256 positions a plane), sliding along z.  x is the caller's and may start at any
// float: ALIGNED (to 16 bytes) copies it four floats at a time, otherwise one.
struct Wgrad0 {
  static constexpr int TILE = 18 * 18 * 16, STEP = TILE + 4096;  // padded planes and rows of one sample, its gradients
  static constexpr size_t SMEM = sizeof(float) * kRing * STEP;
};
template <bool ALIGNED>
__global__ void __launch_bounds__(256, 1) conv0_bwd_param_kernel(int N, const float* __restrict__ dy,
                                                                 const float* __restrict__ x, float* __restrict__ gW,
                                                                 float* __restrict__ gb) {
  extern __shared__ __align__(16) float sm[];
  const int tid = threadIdx.x, co = blockIdx.x / 3, ky = blockIdx.x % 3, ox = tid & 15, oy = tid >> 4;
  for (int e = tid; e < kRing * Wgrad0::STEP; e += 256) sm[e] = 0.f;
  __syncthreads();
  auto stage = [&](int slot, int n) {
    float* t = sm + slot * Wgrad0::STEP;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int e = tid + 256 * u, c = 4 * (e & 3), ry = (e >> 2) & 15, rz = e >> 6;
      float* xd = t + ((rz + 1) * 18 + ry + 1) * 16 + c;
      const float* xs = x + ((int64_t)n << 12) + 4 * e;
      if (ALIGNED) cp16(xd, xs, true);
      else cp16_by_float(xd, xs);
      cp16(t + Wgrad0::TILE + 4 * e, dy + (((int64_t)n * 16 + co) << 12) + 4 * e, true);
    }
  };
  float acc[10];  // [kz][kx], then the bias
#pragma unroll
  for (int k = 0; k < 10; ++k) acc[k] = 0.f;
#pragma unroll
  for (int p = 0; p < kRing - 1; ++p) {
    if (p < N) stage(p, p);
    cp_commit();
  }
  const int left = ox > 0 ? -1 : 0, right = ox < 15 ? 1 : 0;
  for (int n = 0; n < N; ++n) {
    cp_wait<kRing - 2>();
    __syncthreads();
    if (n + kRing - 1 < N) stage((n + kRing - 1) % kRing, n + kRing - 1);
    cp_commit();
    const float* t = sm + (n % kRing) * Wgrad0::STEP;
    const float* b = t + (oy + ky) * 16 + ox;
    const float* d = t + Wgrad0::TILE + tid;
    auto row = [&](int z, float (&w)[3]) {
      const float* p = b + z * 288;
      const float l = p[left], r = p[right];
      w[0] = ox > 0 ? l : 0.f;
      w[1] = p[0];
      w[2] = ox < 15 ? r : 0.f;
    };
    float w[3][3];
    row(0, w[1]);
    row(1, w[2]);
#pragma unroll
    for (int z = 0; z < 16; ++z) {
#pragma unroll
      for (int kx = 0; kx < 3; ++kx) {
        w[0][kx] = w[1][kx];
        w[1][kx] = w[2][kx];
      }
      row(z + 2, w[2]);
      const float dz = d[256 * z];
#pragma unroll
      for (int k = 0; k < 9; ++k) acc[k] = fmaf(dz, w[k / 3][k % 3], acc[k]);
      acc[9] += dz;
    }
  }
  cp_wait<0>();
  block_tree_256<10>(acc, sm);
  if (tid == 0) {
#pragma unroll
    for (int k = 0; k < 9; ++k) gW[co * 27 + (k / 3) * 9 + ky * 3 + k % 3] = acc[k];
    if (ky == 0) gb[co] = acc[9];
  }
}

// head: g = mean of the last activation, z = [g, feats], logits, softmax,
// per-sample cross-entropy (labels may be null); one warp per sample, a lane per
// channel, then a lane per class
__global__ void __launch_bounds__(128) head_fwd_kernel(int N, const float* __restrict__ a4,
                                                       const float* __restrict__ feats, const float* __restrict__ wfc,
                                                       const float* __restrict__ bfc,
                                                       const int32_t* __restrict__ labels, float* __restrict__ z,
                                                       float* __restrict__ prob, float* __restrict__ out_prob,
                                                       float* __restrict__ loss_n) {
  __shared__ float zs[4][kZ];
  const int wid = threadIdx.x >> 5, n = blockIdx.x * 4 + wid, lane = threadIdx.x & 31;
  if (n >= N) return;
  const float4* a = reinterpret_cast<const float4*>(a4 + ((int64_t)n * kHidden + lane) * 8);
  const float4 u = a[0], v = a[1];
  float s8 = 0.f;
  s8 += u.x;
  s8 += u.y;
  s8 += u.z;
  s8 += u.w;
  s8 += v.x;
  s8 += v.y;
  s8 += v.z;
  s8 += v.w;
  zs[wid][lane] = s8 * 0.125f;
  if (lane < kFeat) zs[wid][kHidden + lane] = feats[kFeat * n + lane];
  __syncwarp();
  z[n * kZ + lane] = zs[wid][lane];
  if (lane < kFeat) z[n * kZ + kHidden + lane] = zs[wid][kHidden + lane];
  float lk = 0.f;
  if (lane < kClass) {
    lk = bfc[lane];
#pragma unroll
    for (int j = 0; j < kZ; ++j) lk = fmaf(wfc[lane * kZ + j], zs[wid][j], lk);
  }
  float lg[kClass], mx = -INFINITY;
#pragma unroll
  for (int k = 0; k < kClass; ++k) {
    lg[k] = __shfl_sync(0xffffffffu, lk, k);
    mx = fmaxf(mx, lg[k]);
  }
  if (lane != 0) return;
  float den = 0.f;
#pragma unroll
  for (int k = 0; k < kClass; ++k) den += expf(lg[k] - mx);
#pragma unroll
  for (int k = 0; k < kClass; ++k) {
    const float p = expf(lg[k] - mx) / den;
    prob[n * kClass + k] = p;
    if (out_prob) out_prob[n * kClass + k] = p;
  }
  if (labels) {
    // a label outside the rungs gives a NaN loss (and no one-hot term in the gradient)
    const int lab = labels[n];
    float l = NAN;
#pragma unroll
    for (int k = 0; k < kClass; ++k)
      if (k == lab) l = -(lg[k] - mx - logf(den));
    loss_n[n] = l;
  }
}

// Backward of the head: blocks below ndata make d4 = (dz / 8) broadcast over the 8
// positions, masked by the last ReLU; the last block adds the dense layer's
// gradients and the loss over the samples in order, a thread per parameter, from
// samples staged 64 at a time.
constexpr int kHeadChunk = 64;
__global__ void __launch_bounds__(256) head_bwd_kernel(int N, int ndata, const float* __restrict__ prob,
                                                       const int32_t* __restrict__ labels, const float* __restrict__ z,
                                                       const float* __restrict__ wfc, const float* __restrict__ a4,
                                                       const float* __restrict__ loss_n, float* __restrict__ d4,
                                                       float* __restrict__ gWfc, float* __restrict__ gbfc,
                                                       float* __restrict__ loss) {
  const float invN = 1.f / (float)N;
  if ((int)blockIdx.x < ndata) {
    const int idx = blockIdx.x * 256 + threadIdx.x;  // (n, channel)
    if (idx >= N * kHidden) return;
    const int n = idx / kHidden, c = idx % kHidden;
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < kClass; ++k)
      s = fmaf((prob[n * kClass + k] - (labels[n] == k ? 1.f : 0.f)) * invN, wfc[k * kZ + c], s);
    s *= 0.125f;
    const float4* a = reinterpret_cast<const float4*>(a4 + (int64_t)idx * 8);
    float4* d = reinterpret_cast<float4*>(d4 + (int64_t)idx * 8);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float4 m = a[h];
      d[h] = make_float4(m.x > 0.f ? s : 0.f, m.y > 0.f ? s : 0.f, m.z > 0.f ? s : 0.f, m.w > 0.f ? s : 0.f);
    }
    return;
  }
  __shared__ float ts[kHeadChunk][kClass], zs[kHeadChunk][kZ], ls[kHeadChunk];
  const int p = threadIdx.x;
  const int k = p < kClass * kZ ? p / kZ : p - kClass * kZ, j = p % kZ;
  float s = 0.f;
  for (int n0 = 0; n0 < N; n0 += kHeadChunk) {
    const int cnt = min(kHeadChunk, N - n0);
    __syncthreads();
    for (int e = p; e < cnt * kClass; e += 256) {
      const int n = n0 + e / kClass, c = e % kClass;
      ts[e / kClass][c] = (prob[n * kClass + c] - (labels[n] == c ? 1.f : 0.f)) * invN;
    }
    for (int e = p; e < cnt * kZ; e += 256) zs[e / kZ][e % kZ] = z[n0 * kZ + e];
    if (p < cnt) ls[p] = loss_n[n0 + p];
    __syncthreads();
    if (p < kClass * kZ) {
      for (int n = 0; n < cnt; ++n) s = fmaf(ts[n][k], zs[n][j], s);
    } else if (p < kClass * kZ + kClass) {
      for (int n = 0; n < cnt; ++n) s += ts[n][k];
    } else if (p == kClass * kZ + kClass) {
      for (int n = 0; n < cnt; ++n) s += ls[n];
    }
  }
  if (p < kClass * kZ) gWfc[p] = s;
  else if (p < kClass * kZ + kClass) gbfc[p - kClass * kZ] = s;
  else if (p == kClass * kZ + kClass) *loss = s / (float)N;
}

__global__ void adam_kernel(int n, float* __restrict__ theta, const float* __restrict__ g, float* __restrict__ m,
                            float* __restrict__ v, float lr, float b1, float b2, float eps, float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.f - b1) * gi;
  const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  theta[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// adaptive average pooling of one density field (element order (i*ny + j)*nz + k)
// to 16^3: window i covers [floor(i*n/16), ceil((i+1)*n/16)) along each axis
__global__ void pool16_kernel(int nx, int ny, int nz, const double* __restrict__ d, float* __restrict__ out) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= kVox) return;
  const int c = idx % kS0, b = (idx / kS0) % kS0, a = idx / (kS0 * kS0);
  const int x0 = a * nx / kS0, x1 = ((a + 1) * nx + kS0 - 1) / kS0;
  const int y0 = b * ny / kS0, y1 = ((b + 1) * ny + kS0 - 1) / kS0;
  const int z0 = c * nz / kS0, z1 = ((c + 1) * nz + kS0 - 1) / kS0;
  double s = 0.0;
  for (int i = x0; i < x1; ++i)
    for (int j = y0; j < y1; ++j)
      for (int k = z0; k < z1; ++k) s += d[((int64_t)i * ny + j) * nz + k];
  out[idx] = (float)(s / ((double)(x1 - x0) * (y1 - y0) * (z1 - z0)));
}

}  // namespace
}  // namespace simpfem

using namespace simpfem;

struct simpfem_cnn {
  int max_batch = 0;
  int64_t step = 0;
  DevBuf theta, wpack, grad, m, v;  // wpack: the forward layout, then the data-gradient one
  DevBuf act[5];   // act[0] unused (the input is the caller's), act[1..4] layer outputs
  DevBuf dact[5];  // gradients of the layer outputs act[1..4] (dact[0] unused)
  DevBuf z, prob, loss_n, loss;
};

namespace {

// layer shapes of the kernels' templates: channels and planes per block, channels
// and positions per thread
using F1 = ConvS2<16, 16, 16, 16, 1, 2, 2>;
using F2 = ConvS2<16, 32, 8, 16, 2, 2, 2>;
using F3 = ConvS2<32, 32, 4, 8, 2, 1, 1>;
using D1 = DgradS2<16, 16, 16, 4, 1, 4>;
using D2 = DgradS2<16, 32, 8, 4, 2, 1>;
using D3 = DgradS2<32, 32, 4, 2, 4, 1>;
using G1 = WgradS2<16, 16, 16, 24>;
using G2 = WgradS2<16, 32, 8, 12>;
using G3 = WgradS2<32, 32, 4, 4>;

template <class K>
void big_smem(K kernel, size_t bytes) {
  SF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
}

void set_attributes() {
  static std::atomic<uint64_t> done;
  SF_CUDA(once_per_device(done, [] {
    big_smem(conv_s2_fwd_kernel<16, 16, 16, 16, 1, 2, 2>, F1::SMEM);
    big_smem(conv_s2_fwd_kernel<16, 32, 8, 16, 2, 2, 2>, F2::SMEM);
    big_smem(conv_s2_fwd_kernel<32, 32, 4, 8, 2, 1, 1>, F3::SMEM);
    big_smem(conv_s2_bwd_data_kernel<16, 16, 16, 4, 1, 4>, D1::SMEM);
    big_smem(conv_s2_bwd_data_kernel<16, 32, 8, 4, 2, 1>, D2::SMEM);
    big_smem(conv_s2_bwd_data_kernel<32, 32, 4, 2, 4, 1>, D3::SMEM);
    big_smem(conv_s2_bwd_param_kernel<16, 16, 16, 24>, G1::SMEM);
    big_smem(conv_s2_bwd_param_kernel<16, 32, 8, 12>, G2::SMEM);
    big_smem(conv_s2_bwd_param_kernel<32, 32, 4, 4>, G3::SMEM);
    big_smem(conv0_bwd_param_kernel<true>, Wgrad0::SMEM);
    big_smem(conv0_bwd_param_kernel<false>, Wgrad0::SMEM);
    return cudaSuccess;
  }));
}

void forward(simpfem_cnn* h, const float* x, const float* feats, const int32_t* labels, int N, float* prob,
             cudaStream_t s) {
  const float* wf = h->wpack.as<float>();
  const float* th = h->theta.as<float>();
  pack_weights_kernel<<<div_up(kParams, 256), 256, 0, s>>>(th, h->wpack.as<float>(), h->wpack.as<float>() + kFwdPad);
  conv0_fwd_kernel<<<16 * N, kC0Threads, 0, s>>>(x, wf, th + b_off(0), h->act[1].as<float>());
  SF_CUDA(sf_launched(2));
  conv_s2_fwd_kernel<16, 16, 16, 16, 1, 2, 2><<<F1::BLOCKS * N, F1::THREADS, F1::SMEM, s>>>(
      h->act[1].as<float>(), wf + f_off(1), th + b_off(1), h->act[2].as<float>());
  SF_CUDA(sf_launched(1));
  conv_s2_fwd_kernel<16, 32, 8, 16, 2, 2, 2><<<F2::BLOCKS * N, F2::THREADS, F2::SMEM, s>>>(h->act[2].as<float>(), wf + f_off(2),
                                                                         th + b_off(2), h->act[3].as<float>());
  SF_CUDA(sf_launched(1));
  conv_s2_fwd_kernel<32, 32, 4, 8, 2, 1, 1><<<F3::BLOCKS * N, F3::THREADS, F3::SMEM, s>>>(h->act[3].as<float>(), wf + f_off(3),
                                                                          th + b_off(3), h->act[4].as<float>());
  SF_CUDA(sf_launched(1));
  head_fwd_kernel<<<div_up(N, 4), 128, 0, s>>>(N, h->act[4].as<float>(), feats, wf + f_off(4), th + b_off(4), labels,
                                               h->z.as<float>(), h->prob.as<float>(), prob, h->loss_n.as<float>());
  SF_CUDA(sf_launched(1));
}

void backward(simpfem_cnn* h, const float* x, const int32_t* labels, int N, cudaStream_t s) {
  float* g = h->grad.as<float>();
  const float* wf = h->wpack.as<float>();
  const float* wb = wf + kFwdPad;
  const int nd = div_up(N * kHidden, 256);
  head_bwd_kernel<<<nd + 1, 256, 0, s>>>(
      N, nd, h->prob.as<float>(), labels, h->z.as<float>(), wf + f_off(4), h->act[4].as<float>(),
      h->loss_n.as<float>(), h->dact[4].as<float>(), g + w_off(4), g + b_off(4), h->loss.as<float>());
  SF_CUDA(sf_launched(1));
  conv_s2_bwd_param_kernel<32, 32, 4, 4><<<cin(3) * cout(3) / 4, 256, G3::SMEM, s>>>(
      N, h->dact[4].as<float>(), h->act[3].as<float>(), g + w_off(3), g + b_off(3));
  SF_CUDA(sf_launched(1));
  conv_s2_bwd_data_kernel<32, 32, 4, 2, 4, 1><<<dim3(div_up(N, 4), 1), D3::THREADS, D3::SMEM, s>>>(
      N, h->dact[4].as<float>(), wb + t_off(3), h->act[3].as<float>(), h->dact[3].as<float>());
  SF_CUDA(sf_launched(1));
  conv_s2_bwd_param_kernel<16, 32, 8, 12><<<cin(2) * cout(2) / 4, 256, G2::SMEM, s>>>(
      N, h->dact[3].as<float>(), h->act[2].as<float>(), g + w_off(2), g + b_off(2));
  SF_CUDA(sf_launched(1));
  conv_s2_bwd_data_kernel<16, 32, 8, 4, 2, 1><<<dim3(div_up(N, 2), 1), D2::THREADS, D2::SMEM, s>>>(
      N, h->dact[3].as<float>(), wb + t_off(2), h->act[2].as<float>(), h->dact[2].as<float>());
  SF_CUDA(sf_launched(1));
  conv_s2_bwd_param_kernel<16, 16, 16, 24><<<cin(1) * cout(1) / 4, 256, G1::SMEM, s>>>(
      N, h->dact[2].as<float>(), h->act[1].as<float>(), g + w_off(1), g + b_off(1));
  SF_CUDA(sf_launched(1));
  conv_s2_bwd_data_kernel<16, 16, 16, 4, 1, 4><<<dim3(N, 4), D1::THREADS, D1::SMEM, s>>>(
      N, h->dact[2].as<float>(), wb + t_off(1), h->act[1].as<float>(), h->dact[1].as<float>());
  SF_CUDA(sf_launched(1));
  auto first = (uintptr_t)x % 16 == 0 ? conv0_bwd_param_kernel<true> : conv0_bwd_param_kernel<false>;
  first<<<48, 256, Wgrad0::SMEM, s>>>(N, h->dact[1].as<float>(), x, g + w_off(0), g + b_off(0));
  SF_CUDA(sf_launched(1));
}

void check_batch(simpfem_cnn* h, int N) {
  if (N < 1 || N > h->max_batch) throw InvalidArg{"simpfem_cnn: batch size outside [1, max_batch]"};
}

}  // namespace

#define CNN_API_BEGIN try {
#define CNN_API_END                         \
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

int simpfem_cnn_n_params(void) { return kParams; }

int simpfem_cnn_create(int max_batch, simpfem_cnn** out) {
  CNN_API_BEGIN
  if (!out || max_batch < 1 || max_batch > 65536) throw InvalidArg{"simpfem_cnn_create: bad argument"};
  auto* h = new simpfem_cnn();
  try {
    h->max_batch = max_batch;
    h->theta.alloc(4 * kParams);
    h->wpack.alloc(4 * (kFwdPad + kBwdWords));
    set_attributes();
    h->grad.alloc(4 * kParams);
    h->m.alloc(4 * kParams);
    h->v.alloc(4 * kParams);
    SF_CUDA(cudaMemset(h->theta.p, 0, 4 * kParams));
    SF_CUDA(cudaMemset(h->grad.p, 0, 4 * kParams));
    SF_CUDA(cudaMemset(h->m.p, 0, 4 * kParams));
    SF_CUDA(cudaMemset(h->v.p, 0, 4 * kParams));
    for (int l = 0; l < 4; ++l) {
      const size_t sz = 4 * (size_t)max_batch * cout(l) * sout(l) * sout(l) * sout(l);
      h->act[l + 1].alloc(sz);
      h->dact[l + 1].alloc(sz);
    }
    h->z.alloc(4 * (size_t)max_batch * kZ);
    h->prob.alloc(4 * (size_t)max_batch * kClass);
    h->loss_n.alloc(4 * (size_t)max_batch);
    h->loss.alloc(4);
  } catch (...) {
    delete h;
    throw;
  }
  *out = h;
  CNN_API_END
}

int simpfem_cnn_destroy(simpfem_cnn* h) {
  delete h;
  return SIMPFEM_OK;
}

int simpfem_cnn_set_params(simpfem_cnn* h, const float* host, int n) {
  CNN_API_BEGIN
  if (!h || !host || n != kParams) throw InvalidArg{"simpfem_cnn_set_params: bad argument"};
  SF_CUDA(cudaMemcpy(h->theta.p, host, 4 * (size_t)n, cudaMemcpyHostToDevice));
  SF_CUDA(cudaMemset(h->m.p, 0, 4 * kParams));
  SF_CUDA(cudaMemset(h->v.p, 0, 4 * kParams));
  h->step = 0;
  CNN_API_END
}

int simpfem_cnn_get_params(simpfem_cnn* h, float* host, int n) {
  CNN_API_BEGIN
  if (!h || !host || n != kParams) throw InvalidArg{"simpfem_cnn_get_params: bad argument"};
  SF_CUDA(cudaMemcpy(host, h->theta.p, 4 * (size_t)n, cudaMemcpyDeviceToHost));
  CNN_API_END
}

int simpfem_cnn_pool16(int nx, int ny, int nz, const double* density, float* out, void* stream) {
  CNN_API_BEGIN
  if (nx < 1 || ny < 1 || nz < 1 || !density || !out) throw InvalidArg{"simpfem_cnn_pool16: bad argument"};
  if ((int64_t)nx * ny * nz > (int64_t)1 << 31 || (int64_t)(nx + 1) * kS0 > INT32_MAX)
    throw InvalidArg{"simpfem_cnn_pool16: grid too large"};
  pool16_kernel<<<div_up(kVox, 256), 256, 0, (cudaStream_t)stream>>>(nx, ny, nz, density, out);
  SF_CUDA(sf_launched(1));
  CNN_API_END
}

int simpfem_cnn_forward(simpfem_cnn* h, const float* x, const float* feats, int N, float* prob, void* stream) {
  CNN_API_BEGIN
  if (!h || !x || !feats || !prob) throw InvalidArg{"simpfem_cnn_forward: null argument"};
  check_batch(h, N);
  cudaStream_t s = (cudaStream_t)stream;
  forward(h, x, feats, nullptr, N, prob, s);
  CNN_API_END
}

int simpfem_cnn_loss_grad(simpfem_cnn* h, const float* x, const float* feats, const int32_t* labels, int N,
                          float* grad_host, float* loss_host, void* stream) {
  CNN_API_BEGIN
  if (!h || !x || !feats || !labels) throw InvalidArg{"simpfem_cnn_loss_grad: null argument"};
  check_batch(h, N);
  cudaStream_t s = (cudaStream_t)stream;
  forward(h, x, feats, labels, N, nullptr, s);
  backward(h, x, labels, N, s);
  if (loss_host) SF_CUDA(cudaMemcpyAsync(loss_host, h->loss.p, 4, cudaMemcpyDeviceToHost, s));
  if (grad_host) SF_CUDA(cudaMemcpyAsync(grad_host, h->grad.p, 4 * (size_t)kParams, cudaMemcpyDeviceToHost, s));
  if (loss_host || grad_host) SF_CUDA(cudaStreamSynchronize(s));
  CNN_API_END
}

int simpfem_cnn_adam_step(simpfem_cnn* h, float lr, float beta1, float beta2, float eps, void* stream) {
  CNN_API_BEGIN
  if (!h) throw InvalidArg{"simpfem_cnn_adam_step: null handle"};
  h->step += 1;
  const float c1 = 1.f - powf(beta1, (float)h->step), c2 = 1.f - powf(beta2, (float)h->step);
  adam_kernel<<<div_up(kParams, 256), 256, 0, (cudaStream_t)stream>>>(
      kParams, h->theta.as<float>(), h->grad.as<float>(), h->m.as<float>(), h->v.as<float>(), lr, beta1, beta2, eps, c1,
      c2);
  SF_CUDA(sf_launched(1));
  CNN_API_END
}

}  // extern "C"
