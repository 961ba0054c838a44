// Detection of the layout of a call's points, and launch of ray-run sampling
// (ray_runs.cuh) of dense float attributes with the trilinear filter.
//
// kDetectRuns finds S from the points themselves, in one launch: a block
// looks at one spot of the array for points where a run starts (the path
// turns back there: the differences before, across and after the start oppose
// each other), takes the most frequent distance between consecutive starts
// beside a few fixed run lengths, and counts, warp by warp, the distinct
// 16x16x2-voxel blocks the 32 points of a warp touch under each candidate.
// The last block to finish adds the counts up and picks the run length; the
// run kernel is used when its warps touch at most 12 blocks (points with no
// locality touch about 32).  Beside it, the blocks count the sort bins of
// their consecutive points, which tells points in no order.
//
// For dense float attributes, whose kernels and grids differ by layout, the
// choice goes to the host through mapped memory on which the call waits: one
// launch and a PCIe write, where clearing counters, copying them back and
// synchronizing the stream held a 14.8M-point call up for 38 us, a third of
// its sampling.  Calls on temporally varying volumes return as soon as their
// kernel is queued: the choice stays in device memory (DeviceLayout), where
// the kernel reads it.
#include <atomic>
#include <chrono>

#include "ray_runs.cuh"

namespace vklcuda {

namespace {

// Candidates: S = 64, 128, 256, 512 and the distance found by the block.
constexpr int kFixed        = 4;
constexpr int kDetectBlocks = 64;
constexpr uint32_t kMinRun  = 8;
constexpr uint64_t kRunSpan = 8 * kMaxRun + 1;  // points a detector block looks at
constexpr float kMaxBlocks  = 12.f;             // distinct blocks per warp of the run kernel, at most
constexpr float kOrderBlocks = 20.f;            // and for any gain from going by rays
constexpr int kDetectWarps  = 8;
// Points are in no order when a spot's kMaxRun consecutive ones fall in more
// than this many of the sort's 1024 bins (random points fill 885, camera-ray
// samples about 170).
constexpr uint32_t kScatteredBins = 600;

// Device scratch: blocks done, the run kernels' error word, the answer for
// the kernels behind the detector, and per block the distinct counts of the
// fixed candidates, of its own, its distance and the bins its points fall in.
struct DetectScratch {
  uint32_t done, error;
  DeviceLayout layout;
  uint32_t counts[kDetectBlocks][kFixed + 3];
};

// What the last block writes to the host: the call's number, last.
struct DetectResult {
  uint32_t S, order, scattered, error, call;
};

// result: nullptr where the host does not ask.
__global__ void __launch_bounds__(32 * kDetectWarps)
    kDetectRuns(const __grid_constant__ DevGrid g, uint64_t n, const float *__restrict__ pts, uint32_t call,
                DetectScratch *__restrict__ scratch, DetectResult *result)
{
  __shared__ uint32_t starts[kMaxRun / 32];
  __shared__ uint32_t hist[kMaxRun];
  __shared__ uint32_t distinct[kFixed + 2];  // per candidate; bins
  __shared__ unsigned long long best;
  __shared__ bool last;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, threads = 32 * kDetectWarps;
  const uint64_t spot = (n - kRunSpan) / kDetectBlocks * blockIdx.x;
  for (uint32_t k = tid; k < kMaxRun; k += threads)
    hist[k] = 0;
  if (tid <= kFixed + 1)
    distinct[tid] = 0;
  if (tid == 0)
    best = 0;
  auto diff = [&](uint64_t i) {
    const float *p = pts + 3 * i;
    return f3{__ldg(p + 3) - __ldg(p), __ldg(p + 4) - __ldg(p + 1), __ldg(p + 5) - __ldg(p + 2)};
  };
  auto opposed = [](f3 a, f3 b) { return a.x * b.x + a.y * b.y + a.z * b.z < 0.f; };
#pragma unroll
  for (uint32_t k = tid; k < kMaxRun; k += threads) {
    const uint64_t i = spot + k + 2;  // starts a run?
    const f3 a = diff(i - 2), b = diff(i - 1), c = diff(i);
    const uint32_t word = __ballot_sync(0xffffffffu, opposed(a, b) && opposed(b, c));
    if (lane == 0)
      starts[k >> 5] = word;
  }
  __syncthreads();
  if (tid < (int)kMaxRun / 32) {
    uint32_t bits = starts[tid];
    while (bits) {
      const uint32_t at = 32 * tid + __ffs(bits) - 1;
      bits &= bits - 1;
      uint32_t v = bits, u = tid;
      while (!v && ++u < kMaxRun / 32)
        v = starts[u];
      if (v)
        atomicAdd(hist + (32 * u + __ffs(v) - 1 - at), 1u);
    }
  }
  __syncthreads();
  // the most frequent distance (the longest of equally frequent ones)
  uint32_t most = 0;
#pragma unroll
  for (uint32_t k = 0; k < kMaxRun / threads; ++k)
    most = max(most, hist[tid + k * threads] << 11 | (tid + k * threads));
  most = __reduce_max_sync(0xffffffffu, most);
  if (lane == 0)
    atomicMax(&best, ((unsigned long long)(most >> 11) << 32) | (most & (kMaxRun - 1)));
  __syncthreads();
  const uint32_t found = (best >> 32) && (uint32_t)best >= kMinRun ? (uint32_t)best : 0u;
#pragma unroll
  for (int c = 0; c <= kFixed; ++c) {
    const uint32_t S = c == kFixed ? found : (64u << c);
    const uint64_t i = spot + (uint64_t)(lane & 7) * S + 4 * warp + (lane >> 3);
    const f3 p       = xfmPoint(g.objectToIndex, f3{__ldg(pts + 3 * i), __ldg(pts + 3 * i + 1), __ldg(pts + 3 * i + 2)});
    const uint32_t same = __match_any_sync(0xffffffffu, tileKey<true>(p));
    const uint32_t d    = __popc(__ballot_sync(0xffffffffu, lane == __ffs(same) - 1));
    if (lane == 0)
      atomicAdd(distinct + c, d);
  }
  __syncthreads();
  for (uint32_t k = tid; k < kSortBins; k += threads)
    hist[k] = 0;
  __syncthreads();
#pragma unroll
  for (uint32_t k = tid; k < kMaxRun; k += threads) {
    const float *x = pts + 3 * (spot + k);
    hist[tileKey<true>(xfmPoint(g.objectToIndex, f3{__ldg(x), __ldg(x + 1), __ldg(x + 2)}))] = 1;
  }
  __syncthreads();
  uint32_t bins = 0;
  for (uint32_t k = tid; k < kSortBins; k += threads)
    bins += hist[k];
  bins = __reduce_add_sync(0xffffffffu, bins);
  if (lane == 0)
    atomicAdd(distinct + kFixed + 1, bins);
  __syncthreads();
  if (tid == 0) {
    uint32_t *out = scratch->counts[blockIdx.x];
    for (int c = 0; c <= kFixed; ++c)
      out[c] = distinct[c];
    out[kFixed + 1] = found;
    out[kFixed + 2] = distinct[kFixed + 1];
    __threadfence();
    last = atomicAdd(&scratch->done, 1u) == kDetectBlocks - 1;
    __threadfence();
  }
  __syncthreads();
  if (!last)
    return;
  // the last block: the distance most blocks found, then the candidate
  // whose warps touch fewest blocks; thread b holds block b's counts
  for (uint32_t k = tid; k < kMaxRun; k += threads)
    hist[k] = 0;
  if (tid <= kFixed + 1)
    distinct[tid] = 0;
  if (tid == 0)
    best = 0;
  uint32_t own[kFixed + 3] = {};
  if (tid < kDetectBlocks) {
#pragma unroll
    for (int c = 0; c < kFixed + 3; ++c)
      own[c] = __ldcg(&scratch->counts[tid][c]);
  }
  __syncthreads();
  if (tid < kDetectBlocks && own[kFixed + 1])
    atomicAdd(hist + own[kFixed + 1], 1u);
  __syncthreads();
  if (tid < kDetectBlocks && own[kFixed + 1])
    atomicMax(&best, ((unsigned long long)hist[own[kFixed + 1]] << 32) | own[kFixed + 1]);
  __syncthreads();
  const uint32_t common = (uint32_t)best, agree = (uint32_t)(best >> 32);
  if (tid < kDetectBlocks) {
#pragma unroll
    for (int c = 0; c <= kFixed; ++c)
      if (c < kFixed || (common && own[kFixed + 1] == common))
        atomicAdd(distinct + c, own[c]);
    atomicAdd(distinct + kFixed + 1, own[kFixed + 2]);
  }
  __syncthreads();
  if (tid == 0) {
    uint32_t S  = 0;
    float least = kOrderBlocks;
    for (int c = 0; c <= kFixed; ++c) {
      const uint32_t blocks = c < kFixed ? kDetectBlocks : agree;
      const float mean      = blocks ? (float)distinct[c] / (float)(blocks * kDetectWarps) : 1e9f;
      if (mean < least || (S == 0 && mean <= least)) {
        least = mean;
        S     = c == kFixed ? common : (64u << c);
      }
    }
    scratch->done         = 0;
    scratch->layout.order = S;
    if (result) {
      result->S         = least <= kMaxBlocks ? S : 0u;
      result->order     = S;
      result->scattered = distinct[kFixed + 1] > kScatteredBins * kDetectBlocks;
      result->error     = scratch->error;
      __threadfence_system();
      *(volatile uint32_t *)&result->call = call;
    }
  }
}

template <class Field, bool GRAD>
void launchRuns(const DevGrid &g, uint64_t n, const float *pts, uint32_t attr, float *out, const RunShape &shape,
                uint32_t *error, cudaStream_t st)
{
  const int fixed = shape.fixedLength();
  const auto k    = fixed == 256   ? kSampleRuns<Field, GRAD, 256>
                    : fixed == 128 ? kSampleRuns<Field, GRAD, 128>
                    : fixed == 64  ? kSampleRuns<Field, GRAD, 64>
                                   : kSampleRuns<Field, GRAD, 0>;
  k<<<(unsigned)shape.tiles(n), kRunThreads, shape.smemBytes(), st>>>(g, n, pts, attr, out, shape, error);
}

DetectScratch *runScratch(RunScratch &scratch, cudaStream_t st)
{
  if (!scratch.counts.ptr) {
    scratch.counts.alloc(sizeof(DetectScratch));
    cudaCheck(cudaMemsetAsync(scratch.counts.ptr, 0, sizeof(DetectScratch), st), "ray-run scratch");
  }
  if (!scratch.result) {
    cudaCheck(cudaHostAlloc(&scratch.result, sizeof(DetectResult), cudaHostAllocMapped | cudaHostAllocPortable),
              "ray-run result");
    *(DetectResult *)scratch.result = DetectResult{};
  }
  return scratch.counts.as<DetectScratch>();
}

}  // namespace

RunScratch::~RunScratch()
{
  if (result)
    cudaFreeHost(result);
}

LayoutSlots::~LayoutSlots()
{
  for (Slot &s : slots)
    if (s.ready)
      cudaEventDestroy(s.ready);
}

bool rayRunsApply(const DevGrid &g, int filter, uint32_t attr)
{
  return g.dense && !g.temporal && filter == kFilterLinear && g.type[attr] == kFloat;
}

PointLayout detectLayout(const DevGrid &g, uint64_t n, const float *pts, RunScratch &scratch, cudaStream_t st)
{
  if (n < 2 * kRunSpan)
    return {};
  DetectScratch *dev = runScratch(scratch, st);
  void *mapped       = nullptr;
  cudaCheck(cudaHostGetDevicePointer(&mapped, scratch.result, 0), "ray-run result");
  const uint32_t call = ++scratch.calls;
  kDetectRuns<<<kDetectBlocks, 32 * kDetectWarps, 0, st>>>(g, n, pts, call, dev, (DetectResult *)mapped);
  cudaCheck(cudaGetLastError(), "ray-run detection launch");
  // The stream's earlier work runs first; a wait of more than a few
  // milliseconds is left to the driver (which also reports a failed launch).
  const volatile DetectResult *r = (const volatile DetectResult *)scratch.result;
  const auto limit               = std::chrono::steady_clock::now() + std::chrono::milliseconds(5);
  for (uint32_t spin = 0; r->call != call; ++spin)
    if ((spin & 255u) == 255u && std::chrono::steady_clock::now() > limit) {
      cudaCheck(cudaStreamSynchronize(st), "ray-run detection");
      break;
    }
  std::atomic_thread_fence(std::memory_order_acquire);
  if (r->error) {
    // a ray-run launch since the last detection gave up waiting for its
    // point copy (its CTAs returned without writing their results)
    cudaCheck(cudaMemsetAsync(&dev->error, 0, 4, st), "ray-run error reset");
    fail("a ray-run sampling launch timed out waiting for its point copy; its results are invalid",
         VKL_UNKNOWN_ERROR);
  }
  return {(int)r->S, (int)r->order, r->scattered != 0};
}

int queueLayout(const DevGrid &g, uint64_t n, const float *pts, LayoutSlots &slots, cudaStream_t st,
                PointLayout &layout)
{
  if (n < 2 * kRunSpan)
    return -1;
  int slot = -1;
  uint64_t used = 0;
  {
    std::lock_guard<std::mutex> lock(slots.mutex);
    if (!slots.words.ptr)
      slots.words.alloc(LayoutSlots::kSlots * sizeof(DetectScratch));
    // the stream's own last slot, a new one, the one used longest ago
    uint64_t bestRank = ~uint64_t(0);
    for (int i = 0; i < LayoutSlots::kSlots; ++i) {
      const LayoutSlots::Slot &s = slots.slots[i];
      const uint64_t rank        = s.used && s.stream == st ? 0 : 1 + s.used;
      if (!s.taken && rank < bestRank) {
        bestRank = rank;
        slot     = i;
      }
    }
    if (slot < 0)
      return -1;
    LayoutSlots::Slot &s = slots.slots[slot];
    if (!s.ready)
      cudaCheck(cudaEventCreateWithFlags(&s.ready, cudaEventDisableTiming), "layout slot");
    used     = s.used;
    s.taken  = true;
    s.stream = st;
    s.used   = ++slots.uses;
  }
  DetectScratch *dev = slots.words.as<DetectScratch>() + slot;
  try {
    if (used)
      cudaCheck(cudaStreamWaitEvent(st, slots.slots[slot].ready, 0), "layout slot");
    else
      cudaCheck(cudaMemsetAsync(dev, 0, sizeof(DetectScratch), st), "layout slot");
    kDetectRuns<<<kDetectBlocks, 32 * kDetectWarps, 0, st>>>(g, n, pts, 0, dev, nullptr);
    cudaCheck(cudaGetLastError(), "layout detection launch");
  } catch (...) {
    releaseLayout(slots, slot, st);
    throw;
  }
  layout.device = &dev->layout;
  return slot;
}

void releaseLayout(LayoutSlots &slots, int slot, cudaStream_t st)
{
  // (a failed record leaves an earlier point to wait for; the device is lost then)
  cudaEventRecord(slots.slots[slot].ready, st);
  std::lock_guard<std::mutex> lock(slots.mutex);
  slots.slots[slot].taken = false;
}

void launchSampleRays(const DevGrid &g, uint64_t n, const float *pts, uint32_t attr, float *out, bool grad, int S,
                      RunScratch &scratch, cudaStream_t st)
{
  if (!n)
    return;
  uint32_t *error = &runScratch(scratch, st)->error;
  const RunShape shape((uint32_t)S);
  if (g.atlasTex[attr])
    grad ? launchRuns<AtlasField, true>(g, n, pts, attr, out, shape, error, st)
         : launchRuns<AtlasField, false>(g, n, pts, attr, out, shape, error, st);
  else
    grad ? launchRuns<DenseField<float>, true>(g, n, pts, attr, out, shape, error, st)
         : launchRuns<DenseField<float>, false>(g, n, pts, attr, out, shape, error, st);
  cudaCheck(cudaGetLastError(), "ray-run kernel launch");
}

}  // namespace vklcuda
