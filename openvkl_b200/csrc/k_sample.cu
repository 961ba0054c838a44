// Sampling entry points of the cuda device: dispatch of a call to the
// per-filter instantiations.
#include "sample_kernels.cuh"

namespace vklcuda {

namespace {

// Which calls take one point per thread (sample_direct.cuh) and which the
// sorted tiles.  Up to kDirectPoints everything runs faster direct (16,000
// points: 9.7 -> 6.5 us float, 17.1 -> 6.3 us VDB, 19.7 -> 6.4 us tricubic;
// 600,000: 36 -> 30, 26 -> 20, 67 -> 55 us), but tricubic floats without an
// atlas, whose bricked loads the sort brings together: camera-ray samples up
// to kDirectBricked (262,000 in 40 per ray 51 -> 35 us, 1M 132 -> 160; other
// types 0.8 to 0.93 of the sort's time at 1M).  Of larger calls:
//  - nearest: one voxel per point, nothing for a sort to gain (12M camera-ray
//    samples 138 -> 75 us, random points 283 -> 262 us);
//  - tricubic through an atlas (14.4M camera-ray samples 1004 -> 912 us; by
//    rays 1047); with bricked loads the sort wins (double: 2.10 against 3.04
//    ms);
//  - trilinear, dense float: by rays where the points come by rays (14.8M
//    samples in 40 per ray 202 us sorted, 159 by rays), point by point where
//    they come in no order (10M: 585 -> 547 us), else the sort (12M samples
//    173 us against 283 point by point).  Other types keep the sort, which
//    with the atlas is the fastest form that needs no knowledge of the layout
//    (shorts, 600^3: 17M random points 795 us, 734 direct; camera rays of 12
//    to 96 samples 192 to 228, 159 to 240 by the best of the float kernels for
//    calls that wait for a detector; double, 4.2M camera-ray samples 81 to 182,
//    88 to 180);
//  - trilinear, sparse with a leaf map: direct (59M camera-ray samples 878 ->
//    781 us, by rays 803; 16M random points 990 -> 620 us; stencil blocks,
//    17M points over a 768^3 domain: random 545 us in tiles, 342 direct, camera
//    rays 242 direct; only points that all lie in active leaves are 4 % faster
//    in tiles, 885 against 922 us);
//  - sparse without a leaf map and sparse tricubic keep the tiles.
constexpr uint64_t kDirectPoints  = uint64_t(1) << 20;
constexpr uint64_t kDirectBricked = uint64_t(3) << 17;

bool useDirect(const DevGrid &g, int filter, uint32_t maxDepth, uint64_t n, uint32_t attr, const PointLayout &layout)
{
  const bool bricked = g.dense && filter == kFilterCubic && g.type[attr] == kFloat && !tilesUseAtlas(g, attr);
  if (n < (bricked ? kDirectBricked : kDirectPoints) || filter == kFilterNearest)
    return true;
  // (2.4M random points of shorts 57 -> 49 us, camera rays of bytes even)
  if (g.dense && filter == kFilterLinear && g.type[attr] != kFloat && n < 4 * kDirectPoints)
    return true;
  if (g.dense)
    return filter == kFilterCubic ? tilesUseAtlas(g, attr) : layout.order || layout.scattered;
  return filter == kFilterLinear && leafMapApplies(g, maxDepth);
}

// Which calls for several attributes take the sorted tiles: a tile has a CTA
// work through 1024 points and their attributes one after another, so it needs
// some hundred thousand points to fill the GPU (four float attributes,
// trilinear: 8,192 points 9.2 us with a thread per point, 13.8 in tiles; 65,536
// even; 262,144 camera-ray samples 28 and 19).  Where the tile gathers with
// plain loads it takes longer still (tricubic, double, four attributes: 8,192
// camera-ray samples 37 us and 162; 262,144 172 and 208; 524,288 373 and 310).
bool useTilesM(const DevGrid &g, int filter, uint32_t maxDepth, uint64_t n, uint32_t M, const uint32_t *attrs)
{
  const bool loads = g.dense ? filter == kFilterCubic && !tilesUseAtlas(g, attrs[0])
                             : filter == kFilterCubic || !leafMapApplies(g, maxDepth);
  return sameField(g, M, attrs) && n >= (uint64_t(1) << (loads ? 19 : 18));
}

void dispatch(const DevGrid &g, int filter, uint32_t maxDepth, uint64_t n, const float *pts,
              uint32_t attr, float *out, bool grad, const PointLayout &layout, cudaStream_t st)
{
  if (n == 0)
    return;
  if (useDirect(g, filter, maxDepth, n, attr, layout)) {
    const uint32_t S = g.dense && filter == kFilterLinear ? (uint32_t)layout.order : 0u;
    if (filter == kFilterNearest)
      dispatchDirect<kFilterNearest>(g, maxDepth, n, pts, attr, out, grad, S, st);
    else if (filter == kFilterCubic)
      dispatchDirect<kFilterCubic>(g, maxDepth, n, pts, attr, out, grad, S, st);
    else
      dispatchDirect<kFilterLinear>(g, maxDepth, n, pts, attr, out, grad, S, st);
  } else if (filter == kFilterCubic) {
    dispatchFilter<kFilterCubic>(g, maxDepth, n, pts, attr, out, grad, st);
  } else {
    dispatchFilter<kFilterLinear>(g, maxDepth, n, pts, attr, out, grad, st);
  }
}

}  // namespace
void launchSample(const DevGrid &g, int filter, uint32_t maxDepth, uint64_t n,
                  const float *points, uint32_t M, const uint32_t *attrs, float *out,
                  const PointLayout &layout, cudaStream_t stream)
{
  if (g.temporal) {  // temporally varying data, sampled at time 0
    launchSampleTemporal(g, filter, n, points, nullptr, M, attrs, out, false, layout, stream);
    return;
  }
  if (M == 1) {
    dispatch(g, filter, maxDepth, n, points, attrs[0], out, false, layout, stream);
  } else if (n) {
    AttrList al{};
    al.count = M;
    for (uint32_t m = 0; m < M; ++m)
      al.a[m] = attrs[m];
    if (!useTilesM(g, filter, maxDepth, n, M, attrs))
      launchSampleMixed(g, filter, maxDepth, n, points, al, out, stream);
    else if (filter == kFilterNearest)
      dispatchFilterM<kFilterNearest>(g, maxDepth, n, points, al, out, stream);
    else if (filter == kFilterCubic)
      dispatchFilterM<kFilterCubic>(g, maxDepth, n, points, al, out, stream);
    else
      dispatchFilterM<kFilterLinear>(g, maxDepth, n, points, al, out, stream);
  }
  cudaCheck(cudaGetLastError(), "sample kernel launch");
}

void launchGradient(const DevGrid &g, int filter, uint32_t maxDepth, uint64_t n,
                    const float *points, uint32_t attr, float *out, const PointLayout &layout,
                    cudaStream_t stream)
{
  if (g.temporal) {
    launchSampleTemporal(g, filter, n, points, nullptr, 1, &attr, out, true, layout, stream);
    return;
  }
  dispatch(g, filter, maxDepth, n, points, attr, out, true, layout, stream);
  cudaCheck(cudaGetLastError(), "gradient kernel launch");
}

}  // namespace vklcuda
