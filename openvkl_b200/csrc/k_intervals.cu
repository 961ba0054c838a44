// Batched interval iteration (vklIterateIntervalsN): one lane per ray through
// the whole DDA.
#include "iterate.cuh"
#include "kernels.h"
#include "objects.h"

namespace vklcuda {

namespace {

constexpr int kBlock = 128;
// Resident blocks per SM asked of the compiler for the interval kernel,
// whose DDA state lives in registers (measured on the 1920x1080-ray
// workload): 4 x 128 threads (128 registers) ran fastest; 6 x 128 fits it in
// 80 registers but ran 10 % slower.
constexpr int kIntervalMinBlocks = 4;

__device__ __forceinline__ f3 ld3(const float *p, uint64_t i)
{
  return {__ldg(p + 3 * i), __ldg(p + 3 * i + 1), __ldg(p + 3 * i + 2)};
}

__global__ void __launch_bounds__(kBlock, kIntervalMinBlocks) kIntervals(const __grid_constant__ DevGrid g,
                                                     uint32_t attr, uint32_t depth,
                                                     DevValueRanges vr, uint64_t n,
                                                     const float *__restrict__ orgs,
                                                     const float *__restrict__ dirs,
                                                     const float *__restrict__ tr,
                                                     uint32_t maxPerRay,
                                                     DevInterval *__restrict__ out,
                                                     uint32_t *__restrict__ counts)
{
  const uint64_t r = (uint64_t)blockIdx.x * kBlock + threadIdx.x;
  if (r >= n)
    return;
  IntervalIt it;
  intervalInit(g, depth, ld3(orgs, r), ld3(dirs, r), __ldg(tr + 2 * r), __ldg(tr + 2 * r + 1), it);
  uint32_t c = 0;
  DevInterval iv;
  while (intervalNext(g, attr, vr, it, iv)) {
    if (c < maxPerRay)
      out[r * maxPerRay + c] = iv;
    ++c;
  }
  counts[r] = c;
}

// Dense volumes: a cell's query never changes the DDA's path (the node
// level is always the query depth), so the kernel is compiled per level
// (DdaCell) and the DDA runs ahead of the value range loads.  Each round takes
// kIntervalLookahead steps with their range loads in flight together, then
// applies intervalNext's tests to the cells in order: a non-empty cell whose
// t is not below tMax ends the ray, a spent budget ends it without emitting,
// a non-empty cell emits [t before, min(t after, tMax)].  Steps taken past
// the end of a ray are dropped (their cells are bounds-checked like any
// other).  The intervals are those of intervalNext, in the same order.
//
// A lane's intervals are contiguous in `out`, those of a warp's lanes are
// not: stored one by one, every store instruction touched 30 sectors (13.6
// GB through L2 for 0.9 GB of intervals on 1280x721 rays, and the kernel
// was bound by them and by the instruction fetch of a DDA unrolled for four
// levels).  Each lane collects up to kIvSlots intervals in its row of shared
// memory (odd pitch: the lanes' rows start in distinct banks) and the warp
// writes the rows out together, 8 lanes per ray on sector-aligned words:
// 1280x721 camera rays through 512x500x512 voxels, two value ranges, 96 slots
// per ray: 2.74 -> 0.94 ms.  Bound by instruction issue (2.3 per cycle of
// the SM).
constexpr int kIntervalLookahead = 8;
// 2 on the upper levels, whose cells (4096^3 and 128^3 voxels) a ray
// crosses few of (400,000 rays through 300x280x310 voxels as one cell: 25.3 ->
// 22.6 us with one value range).
template <int L>
constexpr int kLookahead = L < 2 ? 2 : kIntervalLookahead;
constexpr int kIvSlots           = 16;
constexpr int kIvPitch           = kIvSlots * 5 + 1;  // words
constexpr int kIvRanges          = 32;  // value ranges kept in shared memory
constexpr int kIvRegRanges       = 2;   // and in registers (1.12 -> 0.94 ms with the 32-bit cell addresses)
// 5 x 128 threads per SM: what the shared rows allow.
constexpr int kDenseIntervalMinBlocks = 5;

// Writes the warp's collected intervals (nb per lane, rows of kIvPitch words)
// to each lane's next output slot, word offset `at`.
__device__ __forceinline__ void flushIntervals(const float *rows, float *__restrict__ out, uint64_t at, int nb,
                                               int lane)
{
  __syncwarp();
#pragma unroll 1
  for (int pass = 0; pass < 8; ++pass) {
    const int src      = pass * 4 + (lane >> 3);
    const int words    = 5 * __shfl_sync(0xffffffffu, nb, src);
    const uint64_t dst = __shfl_sync(0xffffffffu, at, src);
    const float *row   = rows + src * kIvPitch;
#pragma unroll 1
    for (int w = (lane & 7) - (int)(dst & 7u); w < words; w += 8)
      if (w >= 0)
        out[dst + (uint32_t)w] = row[w];
  }
  __syncwarp();
}

template <int L>
__global__ void __launch_bounds__(kBlock, kDenseIntervalMinBlocks)
    kIntervalsDense(const __grid_constant__ DevGrid g, uint32_t attr, DevValueRanges vr, uint64_t n,
                    const float *__restrict__ orgs, const float *__restrict__ dirs, const float *__restrict__ tr,
                    uint32_t maxPerRay, DevInterval *__restrict__ out, uint32_t *__restrict__ counts)
{
  constexpr int K = kLookahead<L>;
  __shared__ float rowsAll[kBlock * kIvPitch];
  __shared__ float2 sr[kIvRanges];
  const bool rangesShared = vr.numRanges <= kIvRanges;
  if (rangesShared && threadIdx.x < vr.numRanges)
    sr[threadIdx.x] = make_float2(__ldg(vr.ranges + 2 * threadIdx.x), __ldg(vr.ranges + 2 * threadIdx.x + 1));
  __syncthreads();
  // the first ranges in registers, absent ones as NaN, which nothing overlaps
  // (+inf .. -inf would overlap a cell of all values)
  float2 rr[kIvRegRanges];
#pragma unroll
  for (int i = 0; i < kIvRegRanges; ++i)
    rr[i] = rangesShared && (uint32_t)i < vr.numRanges ? sr[i]
                                                       : make_float2(__builtin_nanf(""), __builtin_nanf(""));
  const int lane    = threadIdx.x & 31;
  float *const rows = rowsAll + (threadIdx.x & ~31) * kIvPitch;
  float *const row  = rows + lane * kIvPitch;
  const uint64_t r  = (uint64_t)blockIdx.x * kBlock + threadIdx.x;
  IntervalItT<DdaCell<L>> it;
  it.tMax          = -kPosInf;
  it.nominalDeltaT = 0.f;
  it.budget        = 0;
  it.dda           = DdaCell<L>{};
  if (r < n)
    intervalInit(g, L, ld3(orgs, r), ld3(dirs, r), __ldg(tr + 2 * r), __ldg(tr + 2 * r + 1), it);
  const float tMax = it.tMax;
  const DenseCellRanges<L> cells(g, attr);
  uint32_t c = 0;
  int nb     = 0;
  bool live  = r < n;
  while (__any_sync(0xffffffffu, live)) {
    float t[K + 1];
    float2 v[K];
    uint32_t inside = 0;
    t[0]            = it.dda.t;
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const float2 *p = cells.at(it.dda.id[L][0], it.dda.id[L][1], it.dda.id[L][2]);
      v[j]            = make_float2(0.f, 0.f);
      if (live && p) {
        v[j] = __ldg(p);
        inside |= 1u << j;
      }
      ddaStep(it.dda);
      t[j + 1] = it.dda.t;
    }
#pragma unroll
    for (int j = 0; j < K; ++j) {
      bool overlap = vr.numRanges == 0;
#pragma unroll
      for (int i = 0; i < kIvRegRanges; ++i)
        overlap |= (rr[i].y >= v[j].x) & (rr[i].x <= v[j].y);
      // (most of a short ray's steps are past its end, and their cells would
      // go through all ranges: 40 ranges, one cell, 400,000 rays 79.7 -> 22.1 us)
      if (vr.numRanges > kIvRegRanges && !overlap && live && ((inside >> j) & 1u)) {
        if (rangesShared) {
          for (uint32_t i = kIvRegRanges; i < vr.numRanges; ++i)
            overlap |= (sr[i].y >= v[j].x) & (sr[i].x <= v[j].y);
        } else {
          overlap = rangesOverlap(vr, v[j].x, v[j].y);
        }
      }
      const bool full = overlap && ((inside >> j) & 1u);
      live            = live && t[j] <= tMax && !(full && !(t[j] < tMax)) && it.budget != (uint32_t)j;
      if (live && full) {
        if (c < maxPerRay) {
          float *const e = row + 5 * nb;
          e[0]           = t[j];
          e[1]           = minx(t[j + 1], tMax);
          e[2]           = v[j].x;
          e[3]           = v[j].y;
          e[4]           = it.nominalDeltaT;
          ++nb;
        }
        ++c;
      }
    }
    it.budget -= K;  // a ray whose budget is below K ends within the round
    if (__any_sync(0xffffffffu, nb > kIvSlots - K) || !__any_sync(0xffffffffu, live)) {
      const uint32_t stored = min(c, maxPerRay);
      flushIntervals(rows, (float *)out, 5 * (r * maxPerRay + stored - nb), nb, lane);
      nb = 0;
    }
  }
  if (r < n)
    counts[r] = c;
}

inline unsigned blocksFor(uint64_t n) { return (unsigned)((n + kBlock - 1) / kBlock); }

}  // namespace

void launchIntervals(const DevGrid &g, uint32_t attr, uint32_t depth, DevValueRanges vr,
                     uint64_t n, const float *origins, const float *directions,
                     const float *tRanges, uint32_t maxPerRay, DevInterval *out,
                     uint32_t *counts, cudaStream_t st)
{
  if (!n)
    return;
  if (g.dense) {
    const auto k = depth == 0   ? kIntervalsDense<0>
                   : depth == 1 ? kIntervalsDense<1>
                   : depth == 2 ? kIntervalsDense<2>
                                : kIntervalsDense<3>;
    k<<<blocksFor(n), kBlock, 0, st>>>(g, attr, vr, n, origins, directions, tRanges, maxPerRay, out, counts);
  } else {
    kIntervals<<<blocksFor(n), kBlock, 0, st>>>(g, attr, depth, vr, n, origins, directions, tRanges, maxPerRay,
                                                 out, counts);
  }
  cudaCheck(cudaGetLastError(), "interval kernel launch");
}

}  // namespace vklcuda
