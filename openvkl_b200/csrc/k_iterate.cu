// Per-call iterator kernels of the cuda device: they back the C API's
// stateful vklIterateInterval / vklIterateHit by advancing a state struct
// that lives in the caller's buffer by one step (the batched forms are in
// k_intervals.cu and k_hits.cu).  Also the batched hit kernel of any voxel
// type and filter, which shares their out-of-line sampling dispatch.

// The filters are inlined at many call sites: the fused form of the tricubic
// sums would give every kernel here its registers.
#define VKL_TRICUBIC_PLAIN 1
#include "iterate.cuh"
#include "kernels.h"
#include "objects.h"

namespace vklcuda {

namespace {

constexpr int kBlock = 128;

__device__ __forceinline__ f3 ld3(const float *p, uint64_t i)
{
  return {__ldg(p + 3 * i), __ldg(p + 3 * i + 1), __ldg(p + 3 * i + 2)};
}

// Any voxel type and filter: one ray per thread through the out-of-line
// sampling dispatch.  CTAS per SM: 1 lets the march keep its 242 registers (two
// are resident), 3 has it spill 576 bytes.  Rays that two per SM take at once
// run 1.1 to 1.5 times as long spilled (20,000 rays through 300x280x310 bytes,
// 1 to 20 isovalues); more rays of a march with few isovalues gain from the
// third (200,000 rays, 1 isovalue 8.8 -> 7.3 ms; with 8 even, tricubic 0.85
// times as fast).
template <int CTAS>
__global__ void __launch_bounds__(kBlock, CTAS) kHitsAny(const __grid_constant__ DevGrid g, uint32_t attr, int filter,
                                                   uint32_t depth, DevValueRanges vr, uint32_t numValues,
                                                   const float *__restrict__ values, uint64_t n,
                                                   const float *__restrict__ orgs, const float *__restrict__ dirs,
                                                   const float *__restrict__ tr, uint32_t maxPerRay,
                                                   DevHit *__restrict__ out, uint32_t *__restrict__ counts)
{
  const uint64_t r = (uint64_t)blockIdx.x * kBlock + threadIdx.x;
  if (r >= n)
    return;
  HitIt h;
  hitInit(g, depth, ld3(orgs, r), ld3(dirs, r), __ldg(tr + 2 * r), __ldg(tr + 2 * r + 1), h);
  uint32_t c = 0;
  DevHit hit;
  const AnySampleHook hook{&g, filter, attr, kNumLevels - 1};
  while (c < kMaxHitsPerRay && hitNextWith(g, hook, attr, vr, numValues, values, h, hit)) {
    if (c < maxPerRay)
      out[r * maxPerRay + c] = hit;
    ++c;
  }
  counts[r] = c;
}

struct IntervalIterStateImpl {
  uint32_t attr;
  IntervalIt it;
};
struct HitIterStateImpl {
  uint32_t attr;
  float time;
  HitIt h;
};

__global__ void kIntervalIterInit(const __grid_constant__ DevGrid g, uint32_t attr, uint32_t depth,
                                  const float *ray, IntervalIterStateImpl *s)
{
  s->attr = attr;
  intervalInit(g, depth, {ray[0], ray[1], ray[2]}, {ray[3], ray[4], ray[5]}, ray[6], ray[7], s->it);
}

__global__ void kIntervalIterNext(const __grid_constant__ DevGrid g, DevValueRanges vr,
                                  IntervalIterStateImpl *s, DevInterval *out, int *result)
{
  DevInterval iv;
  const bool ok = intervalNext(g, s->attr, vr, s->it, iv);
  if (ok)
    *out = iv;
  *result = ok ? 1 : 0;
}

__global__ void kHitIterInit(const __grid_constant__ DevGrid g, uint32_t attr, uint32_t depth,
                             const float *ray, HitIterStateImpl *s)
{
  s->attr = attr;
  s->time = ray[8];
  hitInit(g, depth, {ray[0], ray[1], ray[2]}, {ray[3], ray[4], ray[5]}, ray[6], ray[7], s->h);
}

__global__ void kHitIterNext(const __grid_constant__ DevGrid g, int filter, DevValueRanges vr,
                             uint32_t numValues, const float *values, HitIterStateImpl *s,
                             DevHit *out, int *result)
{
  DevHit hit;
  const bool ok = hitNext(g, filter, s->attr, kNumLevels - 1, vr, numValues, values, s->h, hit, s->time);
  if (ok)
    *out = hit;
  *result = ok ? 1 : 0;
}

}  // namespace

void launchHitsAny(const DevGrid &g, uint32_t attr, int filter, uint32_t depth, DevValueRanges vr,
                   uint32_t numValues, const float *values, uint64_t n, const float *origins,
                   const float *directions, const float *tRanges, uint32_t maxPerRay, DevHit *out,
                   uint32_t *counts, cudaStream_t st)
{
  int dev = 0, sms = 0;
  cudaCheck(cudaGetDevice(&dev), "cudaGetDevice");
  cudaCheck(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "attribute");
  const bool many = n > (uint64_t)sms * 2 * kBlock && numValues <= 4 && filter != kFilterCubic;
  const auto k    = many ? kHitsAny<3> : kHitsAny<1>;
  k<<<(unsigned)((n + kBlock - 1) / kBlock), kBlock, 0, st>>>(g, attr, filter, depth, vr, numValues, values, n,
                                                                     origins, directions, tRanges, maxPerRay, out,
                                                                     counts);
  cudaCheck(cudaGetLastError(), "hit kernel launch");
}

size_t intervalIterStateSize() { return sizeof(IntervalIterStateImpl); }
size_t hitIterStateSize() { return sizeof(HitIterStateImpl); }

void launchIntervalIterInit(const DevGrid &g, uint32_t attr, uint32_t depth, const float *ray,
                            void *state, cudaStream_t st)
{
  kIntervalIterInit<<<1, 1, 0, st>>>(g, attr, depth, ray, (IntervalIterStateImpl *)state);
  cudaCheck(cudaGetLastError(), "interval iterator init");
}

void launchIntervalIterNext(const DevGrid &g, DevValueRanges vr, void *state, DevInterval *out,
                            int *result, cudaStream_t st)
{
  kIntervalIterNext<<<1, 1, 0, st>>>(g, vr, (IntervalIterStateImpl *)state, out, result);
  cudaCheck(cudaGetLastError(), "interval iterator step");
}

void launchHitIterInit(const DevGrid &g, uint32_t attr, uint32_t depth, const float *ray,
                       void *state, cudaStream_t st)
{
  kHitIterInit<<<1, 1, 0, st>>>(g, attr, depth, ray, (HitIterStateImpl *)state);
  cudaCheck(cudaGetLastError(), "hit iterator init");
}

void launchHitIterNext(const DevGrid &g, int filter, DevValueRanges vr, uint32_t numValues,
                       const float *values, void *state, DevHit *out, int *result,
                       cudaStream_t st)
{
  kHitIterNext<<<1, 1, 0, st>>>(g, filter, vr, numValues, values, (HitIterStateImpl *)state, out,
                                result);
  cudaCheck(cudaGetLastError(), "hit iterator step");
}

}  // namespace vklcuda
