// Sampling of several attributes that differ in type, or at few points
// (useTilesM, k_sample.cu) (vklComputeSampleMN, VdbSampler.ispc:131-252): one
// point per thread through the run-time dispatch on type and filter.

// Every type and filter is inlined in one kernel, whose registers the fused
// form of the tricubic sums would decide.
#define VKL_TRICUBIC_PLAIN 1
#include "sample_kernels.cuh"

namespace vklcuda {

namespace {

__global__ void __launch_bounds__(kBlock) kSampleM(const __grid_constant__ DevGrid g, int filter,
                                                   uint32_t maxDepth, uint64_t n,
                                                   const float *__restrict__ pts,
                                                   const __grid_constant__ AttrList attrs,
                                                   float *__restrict__ out)
{
  const uint64_t i = (uint64_t)blockIdx.x * kBlock + threadIdx.x;
  if (i >= n)
    return;
  const f3 p = xfmPoint(g.objectToIndex, loadPoint(pts, i));
  for (uint32_t m = 0; m < attrs.count; ++m)
    out[i * attrs.count + m] = sampleIndexAny(g, filter, attrs.a[m], maxDepth, p);
}

}  // namespace

void launchSampleMixed(const DevGrid &g, int filter, uint32_t maxDepth, uint64_t n, const float *points,
                       const AttrList &attrs, float *out, cudaStream_t stream)
{
  kSampleM<<<(unsigned)((n + kBlock - 1) / kBlock), kBlock, 0, stream>>>(g, filter, maxDepth, n, points, attrs, out);
}

}  // namespace vklcuda
