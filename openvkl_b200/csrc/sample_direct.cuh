// Sampling and gradients with one point per thread, as the points come
// (useDirect, k_sample.cu, says which calls).
//
// The sorted tile kernels give a CTA 1024 or 2048 points: a call of a few
// thousand points runs on a handful of SMs, each thread working through 4 or 8
// points behind a sort, and the sort's shared memory and barriers cost more
// than its locality saves wherever a point reads few cache lines.  Each point
// is computed by the same code, so results are the same.
#pragma once
#include "sample_kernels.cuh"

namespace vklcuda {

constexpr int kDirectBlock = 128;

// The point of a thread: point by point, or by rays (S samples each): a block
// takes 16 consecutive samples of 8 neighbouring rays and a warp 4 of each,
// which lie closer together than 32 samples of one ray.
__device__ __forceinline__ bool directPoint(uint32_t S, uint64_t n, uint64_t &i)
{
  if (!S) {
    i = (uint64_t)blockIdx.x * kDirectBlock + threadIdx.x;
    return i < n;
  }
  constexpr uint32_t kSamples = kDirectBlock / 8;
  const uint32_t segs = (S + kSamples - 1) / kSamples, rays = blockIdx.x / segs;
  const uint32_t s = (blockIdx.x - rays * segs) * kSamples + (threadIdx.x >> 3);
  i                = ((uint64_t)rays * 8 + (threadIdx.x & 7u)) * S + s;
  return s < S && i < n;
}
inline unsigned directBlocks(uint32_t S, uint64_t n)
{
  if (!S)
    return (unsigned)((n + kDirectBlock - 1) / kDirectBlock);
  constexpr uint32_t kSamples = kDirectBlock / 8;
  return (unsigned)(((n + S - 1) / S + 7) / 8 * ((S + kSamples - 1) / kSamples));
}

// CTAs of 128 threads per SM: 10 (48 registers) is between the best of camera
// rays and of random points for sparse float leaves (59M camera-ray samples
// over the 1024^3 shells 781 us; 12 CTAs 759, 8 CTAs 809); coded leaves, which
// would spill at 48, take 8 (16.8M points in active leaves, 1536^3 shells:
// FP16 codes 1399 -> 1267 us, 12 CTAs 1590; FP16 blocks 922 -> 910).
template <class Field, int FILTER>
struct DirectTraits {
  static constexpr int kMinBlocks = FILTER == kFilterCubic ? 4 : 10;
};
template <typename T>
struct DirectTraits<MappedField<T>, kFilterLinear> {
  static constexpr int kMinBlocks = LeafCodec<T>::kScaled ? 8 : 10;
};

template <class Field, int FILTER, bool GRAD>
__global__ void __launch_bounds__(kDirectBlock, DirectTraits<Field, FILTER>::kMinBlocks)
    kSampleDirect(const __grid_constant__ DevGrid g, uint32_t maxDepth, uint32_t S, uint64_t n,
                  const float *__restrict__ pts, uint32_t attr, float *__restrict__ out)
{
  uint64_t i;
  if (!directPoint(S, n, i))
    return;
  const float *x = pts + 3 * i;
  const f3 p     = xfmPoint(g.objectToIndex, f3{__ldcs(x), __ldcs(x + 1), __ldcs(x + 2)});
  const Field F  = makeField<Field>(g, attr, maxDepth);
  if constexpr (GRAD) {
    f3 r = {0.f, 0.f, 0.f};
    if constexpr (FILTER == kFilterCubic)
      r = xfmNormal(g.objectToIndex, gradientCubic(F, p));
    else if constexpr (FILTER == kFilterLinear)
      r = xfmNormal(g.objectToIndex, gradientLinear(F, p));
    float *o = out + 3 * i;
    __stcs(o, r.x);
    __stcs(o + 1, r.y);
    __stcs(o + 2, r.z);
  } else {
    __stcs(out + i, filterAt<Field, FILTER>(F, g.constantCellData != 0, p));
  }
}

struct DirectLaunch {
  static constexpr bool kTile = false;
  uint32_t S = 0;  // samples per ray, 0: point by point

  template <class Field, int FILTER>
  void run(const DevGrid &g, uint32_t maxDepth, uint64_t n, const float *pts, uint32_t attr, float *out,
           bool grad, cudaStream_t st) const
  {
    const auto k = grad ? kSampleDirect<Field, FILTER, true> : kSampleDirect<Field, FILTER, false>;
    k<<<directBlocks(S, n), kDirectBlock, 0, st>>>(g, maxDepth, S, n, pts, attr, out);
  }
};

template <int FILTER>
void dispatchDirect(const DevGrid &g, uint32_t maxDepth, uint64_t n, const float *pts,
                    uint32_t attr, float *out, bool grad, uint32_t S, cudaStream_t st)
{
  dispatchTyped<FILTER>(DirectLaunch{S}, g, maxDepth, n, pts, attr, out, grad, st);
}

}  // namespace vklcuda
