// Sums over a whole grid of co-resident blocks (cooperative launches), without
// leaving the kernel.
//
// Every block publishes its part of a sum as two 64-bit words, each holding 32
// bits of the value and the 32-bit number of the exchange; a reader polls the
// words until they carry that number, so a value and its arrival are one load
// and no counter, fence or second read is needed (data and flag in one word, as in the
// low-latency "LL" protocol of NCCL).  Up to kGridFlat blocks each
// block reads all parts; beyond that block 0 reads them and publishes the sum in
// a few copies for the others, because the polls of every block on every part
// load the L2 slices that hold them (one value, with the block-wide sum before
// it: 148 blocks 1.66 us through block 0, 3.7 us all to all, 1.9 us with an
// atomic counter; 8 blocks 1.28, 1.09 and 1.46).  The parts are added in one fixed
// order, so the sum is the same in every block and from run to run.  Slots
// alternate between two halves: a block writes exchange e + 2 only after it has
// seen the sum of e + 1, to which every block adds only after it has read e.
//
// Every wait is bounded: after GridExchange's number of unsuccessful polls the exchange
// reports failure, the block leaves its loop and the others, no longer served,
// do the same; the host reads the flag.  Block 0 keeps the number of the last
// exchange for the next launch on the buffer.  With up to kGridFlat blocks the others
// may have passed an exchange that block 0 gave up and left parts of the next, so
// after a failure it keeps a number beyond any in the slots (grid_last).
#pragma once

#include "common.cuh"

namespace simpfem {

constexpr int kGridSlots = 256;
constexpr int kGridCopies = 8;       // copies of a sum published by block 0
constexpr int kGridMaxBlocks = 160;  // blocks of one exchange: a multiple of 32 (a B200 has 148 SMs)
constexpr int kGridFlat = 32;
constexpr int kGridMaxVals = 4;
// one exchange buffer: [2 halves][kGridMaxVals][kGridSlots] slots of two words
constexpr size_t kGridCommBytes = (size_t)2 * kGridMaxVals * kGridSlots * 16;
static_assert(kGridMaxBlocks + kGridCopies <= kGridSlots, "slots");

// An exchange buffer and how often a block polls it before it gives up (block 0 by
// itself, so that a test can make one side of an exchange give up alone).
struct GridExchange {
  ulonglong2* slots = nullptr;
  unsigned* last = nullptr;  // number of the last exchange
  int polls = kGridPolls, polls0 = kGridPolls;
  __device__ __forceinline__ int limit() const { return blockIdx.x == 0 ? polls0 : polls; }
};

// what *last becomes when block 0 leaves at exchange epoch
__device__ __forceinline__ unsigned grid_last(unsigned epoch, bool ok) { return ok ? epoch : epoch + 2; }

__device__ __forceinline__ void grid_put(ulonglong2* slot, double v, unsigned epoch) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v), e = epoch;
  const unsigned long long lo = (b & 0xffffffffull) | (e << 32), hi = (b >> 32) | (e << 32);
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};\n" ::"l"(slot), "l"(lo), "l"(hi) : "memory");
}

__device__ __forceinline__ bool grid_get(const ulonglong2* slot, double& v, unsigned epoch) {
  unsigned long long lo, hi;
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];\n" : "=l"(lo), "=l"(hi) : "l"(slot) : "memory");
  v = __longlong_as_double((long long)((lo & 0xffffffffull) | (hi << 32)));
  return (unsigned)(lo >> 32) == epoch && (unsigned)(hi >> 32) == epoch;
}

// Sum (or maximum) of NV values per block over the grid, by warp 0 of every
// block (its 32 lanes call this together): v[k] of lane 0 is the block's part; on
// return every lane holds the result.  False when a wait ran out.
template <int NV, bool MAX = false>
__device__ __forceinline__ bool grid_allreduce_warp(const GridExchange& x, unsigned epoch, double (&v)[NV]) {
  const int lane = threadIdx.x & 31, nb = (int)gridDim.x, polls = x.limit();
  ulonglong2* half = x.slots + (size_t)(epoch & 1) * kGridMaxVals * kGridSlots;
#pragma unroll
  for (int k = 0; k < NV; ++k)
    if (lane == 0) grid_put(half + k * kGridSlots + blockIdx.x, v[k], epoch);
  bool all = false;
  if (nb <= kGridFlat || blockIdx.x == 0) {
    constexpr int PER = kGridMaxBlocks / 32;
    double got[NV][PER];
    for (int tries = 0; tries < polls && !all; ++tries) {
      bool ok = true;
#pragma unroll
      for (int k = 0; k < NV; ++k)
#pragma unroll
        for (int p = 0; p < PER; ++p) {
          const int b = lane + 32 * p;
          got[k][p] = MAX ? -INFINITY : 0.0;
          if (b < nb) ok = grid_get(half + k * kGridSlots + b, got[k][p], epoch) && ok;
        }
      all = __all_sync(0xffffffffu, ok);
    }
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      double s = got[k][0];
#pragma unroll
      for (int p = 1; p < PER; ++p) s = MAX ? fmax(s, got[k][p]) : s + got[k][p];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const double t = __shfl_xor_sync(0xffffffffu, s, o);
        s = MAX ? fmax(s, t) : s + t;
      }
      v[k] = s;
      if (all && nb > kGridFlat && lane < kGridCopies) grid_put(half + k * kGridSlots + kGridMaxBlocks + lane, s, epoch);
    }
  } else {
    for (int tries = 0; tries < polls && !all; ++tries) {
      bool ok = true;
#pragma unroll
      for (int k = 0; k < NV; ++k)
        ok = grid_get(half + k * kGridSlots + kGridMaxBlocks + blockIdx.x % kGridCopies, v[k], epoch) && ok;
      all = __all_sync(0xffffffffu, ok);
    }
  }
  return all;
}

// Sum of nparts numbered parts, added one by one in their order, as a kernel with one
// part a block and one thread for the sum adds them.  The caller has put its parts
// into half + number; every lane holds the sum on return.  stage: shared memory of
// kGridParts doubles, 16-byte aligned.
constexpr int kGridParts = 2 * kGridMaxBlocks;
static_assert(kGridParts + kGridCopies <= kGridMaxVals * kGridSlots && kGridParts % 16 == 0, "slots");

__device__ __forceinline__ bool grid_sum_parts_warp(ulonglong2* half, int polls, unsigned epoch, int nparts,
                                                    double* stage, double& v) {
  const int lane = threadIdx.x & 31, nb = (int)gridDim.x;
  bool all = false;
  if (nb <= kGridFlat || blockIdx.x == 0) {
    constexpr int PER = kGridParts / 32;
    for (int tries = 0; tries < polls && !all; ++tries) {
      bool ok = true;
#pragma unroll
      for (int p = 0; p < PER; ++p) {
        const int b = lane + 32 * p;
        double got = 0.0;
        if (b < nparts) ok = grid_get(half + b, got, epoch) && ok;
        stage[b] = got;
      }
      all = __all_sync(0xffffffffu, ok);
    }
    __syncwarp();
    const double s = ordered_sum(stage, nparts);
    __syncwarp();
    v = s;
    if (all && nb > kGridFlat && lane < kGridCopies) grid_put(half + kGridParts + lane, s, epoch);
  } else {
    for (int tries = 0; tries < polls && !all; ++tries)
      all = __all_sync(0xffffffffu, grid_get(half + kGridParts + blockIdx.x % kGridCopies, v, epoch));
  }
  return all;
}

// SMs of the current device (blocks of a cooperative grid at one block per SM).
int grid_sm_count();

}  // namespace simpfem
