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
// stages its operands in shared memory and a thread keeps a tile of outputs in
// registers:
//   forward        4 channels x 2-4 positions a thread, the input channels split over the block
//   data gradient  2 x 2 x 2 input cells (every parity class of the stride: 27 taps per cell),
//                  two cells x 2-4 input channels a thread
//   weight gradient 4 output channels x 1 input channel x 27 taps a thread, sliding
//                  along a row; blocks write partial sums over their samples, one
//                  kernel adds them in block order
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
constexpr int kFwdWords = f_off(4) + kClass * kZ, kBwdWords = t_off(4);
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
template <int CI, int CO, int S, int OZB, int PX, int KS>
struct ConvS2 {
  static constexpr int O = S / 2, P = S + 1, PL = 2 * (OZB - 1) + 3;  // staged planes
  static constexpr int POS = OZB * O * O, TP = POS / PX, TC = CO / 4, TPS = TP * TC;
  static constexpr int THREADS = TPS * KS;
  static constexpr int IN = CI * PL * P * P, W = CI * 27 * CO, RED = KS * CO * POS;
  static constexpr size_t SMEM = sizeof(float) * (((IN + 3) / 4 * 4 > RED ? (IN + 3) / 4 * 4 : RED) + W);
};

template <int CI, int S, int PL>
__device__ __forceinline__ void stage_planes(float* dst, const float* __restrict__ xn, int iz0, int tid, int nt) {
  constexpr int P = S + 1;
  for (int e = tid; e < CI * PL * P * P; e += nt) {
    const int c = e % P, r = (e / P) % P, p = (e / (P * P)) % PL, ci = e / (P * P * PL);
    const int iz = iz0 + p;
    dst[e] = (iz >= 0 && r > 0 && c > 0) ? xn[((ci * S + iz) * S + r - 1) * S + c - 1] : 0.f;
  }
}

template <int CI, int CO, int S, int OZB, int PX, int KS>
__global__ void __launch_bounds__(ConvS2<CI, CO, S, OZB, PX, KS>::THREADS)
    conv_s2_fwd_kernel(const float* __restrict__ x, const float* __restrict__ wf, const float* __restrict__ bias,
                       float* __restrict__ y) {
  using C = ConvS2<CI, CO, S, OZB, PX, KS>;
  extern __shared__ __align__(16) float sm[];
  float* in = sm;
  float* ws = sm + (C::SMEM / sizeof(float) - C::W);
  constexpr int ZB = C::O / OZB;
  const int n = blockIdx.x / ZB, oz0 = (blockIdx.x % ZB) * OZB, tid = threadIdx.x;
  copy_f4(ws, wf, C::W, tid, C::THREADS);
  stage_planes<CI, S, C::PL>(in, x + (int64_t)n * CI * S * S * S, 2 * oz0 - 1, tid, C::THREADS);
  __syncthreads();
  const int ks = tid / C::TPS, t = tid % C::TPS, cq = t % C::TC, pg = t / C::TC;
  constexpr int GX = C::O / PX;
  const int ox = (pg % GX) * PX, oy = (pg / GX) % C::O, oz = pg / (GX * C::O);
  float acc[4][PX];
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int q = 0; q < PX; ++q) acc[c][q] = 0.f;
  for (int ci = ks; ci < CI; ci += KS) {
    const float* base = in + ((ci * C::PL + 2 * oz) * C::P + 2 * oy) * C::P + 2 * ox;
    const float* wb = ws + ci * 27 * CO + 4 * cq;
#pragma unroll
    for (int kz = 0; kz < 3; ++kz)
#pragma unroll
      for (int ky = 0; ky < 3; ++ky) {
        float v[2 * PX + 1];
#pragma unroll
        for (int q = 0; q < 2 * PX + 1; ++q) v[q] = base[(kz * C::P + ky) * C::P + q];
#pragma unroll
        for (int kx = 0; kx < 3; ++kx) {
          const float4 w = *reinterpret_cast<const float4*>(wb + ((kz * 3 + ky) * 3 + kx) * CO);
#pragma unroll
          for (int q = 0; q < PX; ++q) {
            acc[0][q] = fmaf(w.x, v[2 * q + kx], acc[0][q]);
            acc[1][q] = fmaf(w.y, v[2 * q + kx], acc[1][q]);
            acc[2][q] = fmaf(w.z, v[2 * q + kx], acc[2][q]);
            acc[3][q] = fmaf(w.w, v[2 * q + kx], acc[3][q]);
          }
        }
      }
  }
  __syncthreads();  // the input tile becomes the reduction buffer [KS][CO][POS]
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int q = 0; q < PX; ++q) in[(ks * CO + 4 * cq + c) * C::POS + (oz * C::O + oy) * C::O + ox + q] = acc[c][q];
  __syncthreads();
  for (int e = tid; e < CO * C::POS; e += C::THREADS) {
    const int co = e / C::POS, p = e % C::POS;
    float s = bias[co];
#pragma unroll
    for (int k = 0; k < KS; ++k) s += in[k * CO * C::POS + e];
    y[((int64_t)n * CO + co) * C::O * C::O * C::O + oz0 * C::O * C::O + p] = fmaxf(s, 0.f);
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

// Weight and bias gradients of a stride-2 layer: a block adds the contributions
// of its items (an item: OZB output planes of one sample) and writes one partial
// sum of every parameter, weights [co][ci][27] then biases.  A thread holds 4
// output channels x 1 input channel x 27 taps and slides along output rows; PS
// threads of a channel pair share the rows of an item.
template <int CI, int CO, int S, int OZB, int PS>
struct WgradS2 {
  static constexpr int O = S / 2, P = S + 1, PL = 2 * (OZB - 1) + 3, ROWS = OZB * O;
  static constexpr int TPS = CI * CO / 4, THREADS = TPS * PS;
  static constexpr int IN = (CI * PL * P * P + 3) / 4 * 4, DY = ROWS * O * CO;
  static constexpr int NP = CO * CI * 27 + CO;
  static constexpr size_t SMEM = sizeof(float) * ((IN + DY) > (PS > 1 ? NP : 0) ? (IN + DY) : NP);
  static_assert(PS <= ROWS && ROWS % PS == 0, "rows");
};

template <int CI, int CO, int S, int OZB, int PS>
__global__ void __launch_bounds__(WgradS2<CI, CO, S, OZB, PS>::THREADS)
    conv_s2_bwd_param_kernel(int N, const float* __restrict__ dy, const float* __restrict__ x,
                             float* __restrict__ part) {
  using C = WgradS2<CI, CO, S, OZB, PS>;
  extern __shared__ __align__(16) float sm[];
  float* in = sm;            // [CI][PL][P][P]
  float* ds = sm + C::IN;    // [position][CO]
  const int tid = threadIdx.x, ps = tid / C::TPS, t = tid % C::TPS, ci = t % CI, cq = t / CI;
  constexpr int ZB = C::O / OZB, O3 = C::O * C::O * C::O;
  float acc[4][27], bacc[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    bacc[c] = 0.f;
#pragma unroll
    for (int k = 0; k < 27; ++k) acc[c][k] = 0.f;
  }
  const int items = N * ZB;
  for (int it = blockIdx.x; it < items; it += gridDim.x) {
    const int n = it / ZB, oz0 = (it % ZB) * OZB;
    __syncthreads();
    stage_planes<CI, S, C::PL>(in, x + (int64_t)n * CI * S * S * S, 2 * oz0 - 1, tid, C::THREADS);
    for (int e = tid; e < C::DY; e += C::THREADS) {
      const int p = e % (OZB * C::O * C::O), co = e / (OZB * C::O * C::O);
      ds[p * CO + co] = dy[((int64_t)n * CO + co) * O3 + oz0 * C::O * C::O + p];
    }
    __syncthreads();
    for (int row = ps; row < C::ROWS; row += PS) {
      const int oz = row / C::O, oy = row % C::O;
      const float* base = in + ((ci * C::PL + 2 * oz) * C::P + 2 * oy) * C::P;
      const float* drow = ds + row * C::O * CO + 4 * cq;
      float w[9][3];
#pragma unroll
      for (int r = 0; r < 9; ++r) w[r][2] = base[((r / 3) * C::P + r % 3) * C::P];
#pragma unroll
      for (int ox = 0; ox < C::O; ++ox) {
#pragma unroll
        for (int r = 0; r < 9; ++r) {
          const float* b = base + ((r / 3) * C::P + r % 3) * C::P + 2 * ox;
          w[r][0] = w[r][2];
          w[r][1] = b[1];
          w[r][2] = b[2];
        }
        const float4 d = *reinterpret_cast<const float4*>(drow + ox * CO);
        bacc[0] += d.x;
        bacc[1] += d.y;
        bacc[2] += d.z;
        bacc[3] += d.w;
#pragma unroll
        for (int k = 0; k < 27; ++k) {
          const float v = w[k / 3][k % 3];
          acc[0][k] = fmaf(d.x, v, acc[0][k]);
          acc[1][k] = fmaf(d.y, v, acc[1][k]);
          acc[2][k] = fmaf(d.z, v, acc[2][k]);
          acc[3][k] = fmaf(d.w, v, acc[3][k]);
        }
      }
    }
  }
  float* out = part + (int64_t)blockIdx.x * C::NP;
  float* dst = PS > 1 ? sm : out;
  for (int s = 0; s < PS; ++s) {  // the row shares in order
    __syncthreads();
    if (ps == s) {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        float* q = dst + ((4 * cq + c) * CI + ci) * 27;
#pragma unroll
        for (int k = 0; k < 27; ++k) q[k] = s == 0 ? acc[c][k] : q[k] + acc[c][k];
        if (ci == 0) {
          float* b = dst + CO * CI * 27 + 4 * cq + c;
          *b = s == 0 ? bacc[c] : *b + bacc[c];
        }
      }
    }
  }
  if (PS > 1) {
    __syncthreads();
    for (int e = tid; e < C::NP; e += C::THREADS) out[e] = sm[e];
  }
}

// First layer's weight and bias gradients: a thread holds 4 output channels x 27
// taps for one (y, x) of 16 x 4 positions and slides along z; its 64 threads per
// channel quad are then added in a fixed order.
constexpr int kG0Threads = 256, kG0Params = 16 * 27 + 16;
__global__ void __launch_bounds__(kG0Threads) conv0_bwd_param_kernel(int N, const float* __restrict__ dy,
                                                                     const float* __restrict__ x,
                                                                     float* __restrict__ part) {
  __shared__ float in[18 * 18 * 18];
  __shared__ float red[8][4 * 28];
  const int tid = threadIdx.x, lane = tid & 31, cq = tid >> 6, ox = tid & 15, yg = (tid >> 4) & 3;
  float acc[4][28];  // 27 taps, then the bias
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int k = 0; k < 28; ++k) acc[c][k] = 0.f;
  for (int n = blockIdx.x; n < N; n += gridDim.x) {
    __syncthreads();
    for (int e = tid; e < 18 * 18 * 18; e += kG0Threads) {
      const int c = e % 18, r = (e / 18) % 18, p = e / 324;
      const bool ok = c > 0 && c < 17 && r > 0 && r < 17 && p > 0 && p < 17;
      in[e] = ok ? x[((int64_t)n << 12) + ((p - 1) * 16 + r - 1) * 16 + c - 1] : 0.f;
    }
    __syncthreads();
    const float* d0 = dy + (((int64_t)n * 16 + 4 * cq) << 12);
    for (int yy = 0; yy < 4; ++yy) {
      const int oy = 4 * yy + yg;
      float w[3][9];
#pragma unroll
      for (int r = 0; r < 9; ++r) {
        const int q = (oy + r / 3) * 18 + ox + r % 3;
        w[1][r] = in[q];
        w[2][r] = in[324 + q];
      }
#pragma unroll 4
      for (int oz = 0; oz < 16; ++oz) {
#pragma unroll
        for (int r = 0; r < 9; ++r) {
          w[0][r] = w[1][r];
          w[1][r] = w[2][r];
          w[2][r] = in[(oz + 2) * 324 + (oy + r / 3) * 18 + ox + r % 3];
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float d = d0[(c << 12) + (oz * 16 + oy) * 16 + ox];
          acc[c][27] += d;
#pragma unroll
          for (int k = 0; k < 27; ++k) acc[c][k] = fmaf(d, w[k / 9][k % 9], acc[c][k]);
        }
      }
    }
  }
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int k = 0; k < 28; ++k) {
      float s = acc[c][k];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
      if (lane == 0) red[tid >> 5][c * 28 + k] = s;
    }
  __syncthreads();
  float* out = part + (int64_t)blockIdx.x * kG0Params;
  for (int e = tid; e < 16 * 28; e += kG0Threads) {
    const int co = e / 28, k = e % 28, q = co >> 2, j = (co & 3) * 28 + k;
    const float s = red[2 * q][j] + red[2 * q + 1][j];
    if (k < 27) out[co * 27 + k] = s;
    else out[16 * 27 + co] = s;
  }
}

// Partial sums of all four layers added in block order into the gradient.
struct PartSet {
  const float* p[4];
  int blocks[4];
};
__global__ void param_sum_kernel(PartSet ps, float* __restrict__ g) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= w_off(4)) return;
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    const int np = cout(l) * cin(l) * 27 + cout(l), e = i - w_off(l);
    if (e < 0 || e >= np) continue;
    float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
    int b = 0;
    for (; b + 3 < ps.blocks[l]; b += 4) {
      s0 += ps.p[l][(int64_t)b * np + e];
      s1 += ps.p[l][(int64_t)(b + 1) * np + e];
      s2 += ps.p[l][(int64_t)(b + 2) * np + e];
      s3 += ps.p[l][(int64_t)(b + 3) * np + e];
    }
    for (; b < ps.blocks[l]; ++b) s0 += ps.p[l][(int64_t)b * np + e];
    g[i] = (s0 + s1) + (s2 + s3);
  }
}

__device__ __forceinline__ float warp_sum_f(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// head: g = mean of the last activation, z = [g, feats], logits, softmax,
// per-sample cross-entropy (labels may be null); one warp per sample, a lane per
// channel
__global__ void __launch_bounds__(128) head_fwd_kernel(int N, const float* __restrict__ a4,
                                                       const float* __restrict__ feats, const float* __restrict__ wfc,
                                                       const float* __restrict__ bfc,
                                                       const int32_t* __restrict__ labels, float* __restrict__ z,
                                                       float* __restrict__ prob, float* __restrict__ out_prob,
                                                       float* __restrict__ loss_n) {
  const int n = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (n >= N) return;
  const float4* a = reinterpret_cast<const float4*>(a4 + ((int64_t)n * kHidden + lane) * 8);
  const float4 u = a[0], v = a[1];
  const float zz = (((u.x + u.y) + (u.z + u.w)) + ((v.x + v.y) + (v.z + v.w))) * 0.125f;
  const float zf = lane < kFeat ? feats[kFeat * n + lane] : 0.f;
  float lg[kClass], mx = -INFINITY;
#pragma unroll
  for (int k = 0; k < kClass; ++k) {
    float s = wfc[k * kZ + lane] * zz;
    if (lane < kFeat) s = fmaf(wfc[k * kZ + kHidden + lane], zf, s);
    lg[k] = warp_sum_f(s) + bfc[k];
    mx = fmaxf(mx, lg[k]);
  }
  float den = 0.f;
#pragma unroll
  for (int k = 0; k < kClass; ++k) den += expf(lg[k] - mx);
  z[n * kZ + lane] = zz;
  if (lane < kFeat) z[n * kZ + kHidden + lane] = zf;
  if (lane == 0) {
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
}

// Backward of the head: blocks below ndata make d4 = (dz / 8) broadcast over the 8
// positions, masked by the last ReLU; each warp of the others sums one parameter of
// the dense layer (or, the last, the loss) over the samples in a fixed order.
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
  const int p = ((int)blockIdx.x - ndata) * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (p > kClass * kZ + kClass) return;
  float s = 0.f;
  if (p < kClass * kZ) {
    const int k = p / kZ, j = p % kZ;
    for (int n = lane; n < N; n += 32)
      s += ((prob[n * kClass + k] - (labels[n] == k ? 1.f : 0.f)) * invN) * z[n * kZ + j];
  } else if (p < kClass * kZ + kClass) {
    const int k = p - kClass * kZ;
    for (int n = lane; n < N; n += 32) s += (prob[n * kClass + k] - (labels[n] == k ? 1.f : 0.f)) * invN;
  } else {
    for (int n = lane; n < N; n += 32) s += loss_n[n];
  }
  s = warp_sum_f(s);
  if (lane == 0) {
    if (p < kClass * kZ) gWfc[p] = s;
    else if (p < kClass * kZ + kClass) gbfc[p - kClass * kZ] = s;
    else *loss = s / (float)N;
  }
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
  DevBuf theta, wf, wb, grad, m, v;
  DevBuf part[4];  // per-block partial sums of the weight gradients
  DevBuf act[5];   // act[0] unused (the input is the caller's), act[1..4] layer outputs
  DevBuf dact[5];  // gradients of the layer outputs act[1..4] (dact[0] unused)
  DevBuf z, prob, loss_n, loss;
};

namespace {

// layer shapes of the kernels' templates: planes per block, positions a thread,
// splits of the channels or rows over the block
using F1 = ConvS2<16, 16, 16, 1, 4, 4>;
using F2 = ConvS2<16, 32, 8, 4, 4, 4>;
using F3 = ConvS2<32, 32, 4, 2, 2, 16>;
using D1 = DgradS2<16, 16, 16, 4, 1, 4>;
using D2 = DgradS2<16, 32, 8, 4, 2, 1>;
using D3 = DgradS2<32, 32, 4, 2, 4, 1>;
using G1 = WgradS2<16, 16, 16, 1, 4>;
using G2 = WgradS2<16, 32, 8, 4, 2>;
using G3 = WgradS2<32, 32, 4, 2, 1>;

// blocks of a layer's weight-gradient kernel: one per SM, in the last layer one
// per four samples, whose arithmetic is small beside its 27,680 partial sums
int wgrad_blocks(int l, int N) {
  const int sms = 148;
  if (l == 0) return std::min(N, sms);
  if (l == 1) return std::min(8 * N, sms);
  if (l == 2) return std::min(N, sms);
  return std::min((N + 3) / 4, sms / 4);
}
constexpr int wgrad_params(int l) { return cout(l) * cin(l) * 27 + cout(l); }

template <class K>
void big_smem(K kernel, size_t bytes) {
  SF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
}

void set_attributes() {
  static std::atomic<uint64_t> done;
  SF_CUDA(once_per_device(done, [] {
    big_smem(conv_s2_fwd_kernel<16, 16, 16, 1, 4, 4>, F1::SMEM);
    big_smem(conv_s2_fwd_kernel<16, 32, 8, 4, 4, 4>, F2::SMEM);
    big_smem(conv_s2_fwd_kernel<32, 32, 4, 2, 2, 16>, F3::SMEM);
    big_smem(conv_s2_bwd_data_kernel<16, 16, 16, 4, 1, 4>, D1::SMEM);
    big_smem(conv_s2_bwd_data_kernel<16, 32, 8, 4, 2, 1>, D2::SMEM);
    big_smem(conv_s2_bwd_data_kernel<32, 32, 4, 2, 4, 1>, D3::SMEM);
    big_smem(conv_s2_bwd_param_kernel<16, 16, 16, 1, 4>, G1::SMEM);
    big_smem(conv_s2_bwd_param_kernel<16, 32, 8, 4, 2>, G2::SMEM);
    big_smem(conv_s2_bwd_param_kernel<32, 32, 4, 2, 1>, G3::SMEM);
    return cudaSuccess;
  }));
}

void forward(simpfem_cnn* h, const float* x, const float* feats, const int32_t* labels, int N, float* prob,
             cudaStream_t s) {
  const float* wf = h->wf.as<float>();
  const float* th = h->theta.as<float>();
  pack_weights_kernel<<<div_up(kParams, 256), 256, 0, s>>>(th, h->wf.as<float>(), h->wb.as<float>());
  conv0_fwd_kernel<<<16 * N, kC0Threads, 0, s>>>(x, wf, th + b_off(0), h->act[1].as<float>());
  SF_CUDA(sf_launched(2));
  conv_s2_fwd_kernel<16, 16, 16, 1, 4, 4><<<8 * N, F1::THREADS, F1::SMEM, s>>>(
      h->act[1].as<float>(), wf + f_off(1), th + b_off(1), h->act[2].as<float>());
  SF_CUDA(sf_launched(1));
  conv_s2_fwd_kernel<16, 32, 8, 4, 4, 4><<<N, F2::THREADS, F2::SMEM, s>>>(h->act[2].as<float>(), wf + f_off(2),
                                                                         th + b_off(2), h->act[3].as<float>());
  SF_CUDA(sf_launched(1));
  conv_s2_fwd_kernel<32, 32, 4, 2, 2, 16><<<N, F3::THREADS, F3::SMEM, s>>>(h->act[3].as<float>(), wf + f_off(3),
                                                                          th + b_off(3), h->act[4].as<float>());
  SF_CUDA(sf_launched(1));
  head_fwd_kernel<<<div_up(N, 4), 128, 0, s>>>(N, h->act[4].as<float>(), feats, wf + f_off(4), th + b_off(4), labels,
                                               h->z.as<float>(), h->prob.as<float>(), prob, h->loss_n.as<float>());
  SF_CUDA(sf_launched(1));
}

void backward(simpfem_cnn* h, const float* x, const int32_t* labels, int N, cudaStream_t s) {
  float* g = h->grad.as<float>();
  const float* wb = h->wb.as<float>();
  const int nd = div_up(N * kHidden, 256);
  head_bwd_kernel<<<nd + div_up(kClass * kZ + kClass + 1, 8), 256, 0, s>>>(
      N, nd, h->prob.as<float>(), labels, h->z.as<float>(), h->wf.as<float>() + f_off(4), h->act[4].as<float>(),
      h->loss_n.as<float>(), h->dact[4].as<float>(), g + w_off(4), g + b_off(4), h->loss.as<float>());
  SF_CUDA(sf_launched(1));
  PartSet ps;
  for (int l = 0; l < 4; ++l) {
    ps.p[l] = h->part[l].as<float>();
    ps.blocks[l] = wgrad_blocks(l, N);
  }
  conv_s2_bwd_param_kernel<32, 32, 4, 2, 1><<<ps.blocks[3], G3::THREADS, G3::SMEM, s>>>(
      N, h->dact[4].as<float>(), h->act[3].as<float>(), h->part[3].as<float>());
  SF_CUDA(sf_launched(1));
  conv_s2_bwd_data_kernel<32, 32, 4, 2, 4, 1><<<dim3(div_up(N, 4), 1), D3::THREADS, D3::SMEM, s>>>(
      N, h->dact[4].as<float>(), wb + t_off(3), h->act[3].as<float>(), h->dact[3].as<float>());
  SF_CUDA(sf_launched(1));
  conv_s2_bwd_param_kernel<16, 32, 8, 4, 2><<<ps.blocks[2], G2::THREADS, G2::SMEM, s>>>(
      N, h->dact[3].as<float>(), h->act[2].as<float>(), h->part[2].as<float>());
  SF_CUDA(sf_launched(1));
  conv_s2_bwd_data_kernel<16, 32, 8, 4, 2, 1><<<dim3(div_up(N, 2), 1), D2::THREADS, D2::SMEM, s>>>(
      N, h->dact[3].as<float>(), wb + t_off(2), h->act[2].as<float>(), h->dact[2].as<float>());
  SF_CUDA(sf_launched(1));
  conv_s2_bwd_param_kernel<16, 16, 16, 1, 4><<<ps.blocks[1], G1::THREADS, G1::SMEM, s>>>(
      N, h->dact[2].as<float>(), h->act[1].as<float>(), h->part[1].as<float>());
  SF_CUDA(sf_launched(1));
  conv_s2_bwd_data_kernel<16, 16, 16, 4, 1, 4><<<dim3(N, 4), D1::THREADS, D1::SMEM, s>>>(
      N, h->dact[2].as<float>(), wb + t_off(1), h->act[1].as<float>(), h->dact[1].as<float>());
  SF_CUDA(sf_launched(1));
  conv0_bwd_param_kernel<<<ps.blocks[0], kG0Threads, 0, s>>>(N, h->dact[1].as<float>(), x, h->part[0].as<float>());
  param_sum_kernel<<<div_up(w_off(4), 128), 128, 0, s>>>(ps, g);
  SF_CUDA(sf_launched(2));
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
    h->wf.alloc(4 * kFwdWords);
    h->wb.alloc(4 * kBwdWords);
    SF_CUDA(cudaMemset(h->wb.p, 0, 4 * kBwdWords));
    for (int l = 0; l < 4; ++l) h->part[l].alloc(4 * (size_t)wgrad_blocks(l, max_batch) * wgrad_params(l));
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
